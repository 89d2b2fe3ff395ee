"""The work that a user of this framework has it do, as cases that can be prepared, run and timed.

Every case is one pass through the public entry points: the sampling step on host or device logits, a
whole batched generation with the loop control on the device, the LM-head projection with and without
the sampling step behind it, TopK, softmax (with the Multinomial draw behind it) and the cross-entropy
loss with its gradient. Vocabularies are GPT-2's (50,257), Qwen's (151,936) and the 168,320 columns of
the cross-entropy workload; drawn cases take any size from 1,000 columns up to those, odd ones among
them. Logits are seeded normals with peaked columns, the form of gorch_b200/workloads.py, made on the GPU.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from gorch_b200 import generate, row_ops, sampling
from gorch_b200.config import CFG_DTYPE, DTYPE_BF16, DTYPE_F32, MODE_A, MODE_B
from gorch_b200.workloads import GPT2_VOCAB, MIXED_CYCLE, QWEN_VOCAB

CE_VOCAB = 168320
MIN_VOCAB = 1000
MAX_LOGITS_BYTES = 512 * QWEN_VOCAB * 4          # of one sampling, TopK or softmax call
MAX_CE_BYTES = 1500 * CE_VOCAB * 4               # of one cross-entropy call
MAX_WEIGHTS = QWEN_VOCAB * 2048                  # elements of an LM head
MAX_LM_MACS = 512 * QWEN_VOCAB * 1024            # multiply-adds of one projection
TORCH_DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16}
CODES = {"f32": DTYPE_F32, "bf16": DTYPE_BF16}


def _sampling(config: str, temperature: float, top_k: int, top_p: float, mode: int) -> dict:
    """config "rows": every row has these fields; "mixed": MIXED_CYCLE's records in turn, with this mode."""
    return {"config": config, "temperature": temperature, "top_k": top_k, "top_p": top_p, "mode": mode}


def listed() -> list:
    return [
        # The reference's own call: one GPT-2 row in host memory, DefaultGenerateConfig, one id back
        # (model/generate.go:147); what each token of a single user's generation costs beside the forward.
        {"name": "host_row", "kind": "host", "rows": 1, "vocab": GPT2_VOCAB, "sigma": 2.0, "peaks": 16, "peak": 8.0,
         **_sampling("rows", 0.8, 40, 0.0, MODE_A)},
        # A lightly loaded server: few rows, bf16 logits of the Qwen vocabulary, top-k with top-p behind it.
        {"name": "decode_8", "kind": "sample", "rows": 8, "vocab": QWEN_VOCAB, "dtype": "bf16", "sigma": 3.0, "peaks": 32, "peak": 6.0,
         **_sampling("rows", 0.7, 50, 0.95, MODE_B)},
        # Nucleus sampling of a moderate batch, top-k off (the second workload of the benchmark).
        {"name": "nucleus_64", "kind": "sample", "rows": 64, "vocab": GPT2_VOCAB, "dtype": "f32", "sigma": 2.0, "peaks": 16, "peak": 8.0,
         **_sampling("rows", 1.0, 0, 0.9, MODE_A)},
        # Users with settings of their own in one batch: greedy, top-k with top-p, nucleus, wide top-k (the third).
        {"name": "mixed_256", "kind": "sample", "rows": 256, "vocab": GPT2_VOCAB, "dtype": "f32", "sigma": 2.0, "peaks": 16, "peak": 8.0,
         **_sampling("mixed", 0.0, 0, 0.0, MODE_A)},
        # Flat distributions under a deep nucleus: nearly every token takes part (the fourth, the headline).
        {"name": "nucleus_flat_512", "kind": "sample", "rows": 512, "vocab": QWEN_VOCAB, "dtype": "f32", "sigma": 0.25, "peaks": 0, "peak": 0.0,
         **_sampling("rows", 1.0, 0, 0.99, MODE_B)},
        # A large serving batch of bf16 rows with top-k and top-p (the fifth).
        {"name": "topk_1024", "kind": "sample", "rows": 1024, "vocab": QWEN_VOCAB, "dtype": "bf16", "sigma": 3.0, "peaks": 32, "peak": 6.0,
         **_sampling("rows", 0.7, 64, 0.95, MODE_B)},
        # A whole generation of a batch through the generate loop: state, decode steps, polls, results.
        {"name": "generate_16", "kind": "generate", "rows": 16, "vocab": QWEN_VOCAB, "dtype": "bf16", "sigma": 3.0, "peaks": 32, "peak": 6.0,
         "new": 32, **_sampling("rows", 0.7, 50, 0.95, MODE_B)},
        # Hidden states to tokens in one call: the LM head of the Qwen vocabulary under DefaultGenerateConfig.
        {"name": "lm_head_sample_64", "kind": "lm_sample", "rows": 64, "vocab": QWEN_VOCAB, "hidden": 1024,
         **_sampling("rows", 0.8, 40, 0.0, MODE_A)},
        # The projection alone for a large batch, logits kept (scoring, log-probabilities of prompts).
        {"name": "lm_head_logits_512", "kind": "lm_logits", "rows": 512, "vocab": QWEN_VOCAB, "hidden": 1024},
        # TopK wide enough for distillation targets and re-ranking (gorch.TopK, index_ops.go:153).
        {"name": "topk_values_512", "kind": "topk", "rows": 512, "vocab": QWEN_VOCAB, "dtype": "f32", "k": 1000},
        # gorch.Softmax and the gorch.Multinomial draw behind it (index_ops.go:203).
        {"name": "softmax_draw_512", "kind": "softmax", "rows": 512, "vocab": QWEN_VOCAB, "dtype": "f32", "log": False, "draw": True},
        # A training step's loss and gradient on the reference's cross-entropy workload (loss.go:21).
        {"name": "cross_entropy_1500", "kind": "ce", "rows": 1500, "vocab": CE_VOCAB, "dtype": "f32"},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _draw_config(rng, vocab: int) -> dict:
    """Sampling fields in earnest use: greedy, top-k alone or with top-p, a nucleus, plain softmax sampling, a mixed batch."""
    what = rng.choice(["greedy", "top_k", "top_k_top_p", "nucleus", "plain", "mixed"])
    t, mode = round(rng.uniform(0.5, 1.3), 2), rng.choice([MODE_A, MODE_B])
    k, p = _log_int(rng, 5, min(200, vocab // 4)), round(rng.uniform(0.5, 0.99), 3)
    if what == "greedy":
        return _sampling("rows", 0.0, 0, 0.0, MODE_A)
    if what == "mixed":
        return _sampling("mixed", 0.0, 0, 0.0, mode)
    return _sampling("rows", t, k if what.startswith("top_k") else 0, p if what in ("top_k_top_p", "nucleus") else 0.0, mode)


def _draw_spread(rng) -> dict:
    sigma = round(rng.uniform(0.25, 3.0), 2)
    return {"sigma": sigma, "peaks": rng.choice([8, 16, 32]) if sigma >= 1.0 else 0, "peak": round(rng.uniform(4.0, 9.0), 1)}


def draw(rng) -> dict:
    kind = rng.choice(["host", "sample", "sample", "sample", "generate", "lm_sample", "lm_logits", "topk", "softmax", "ce"])
    dtype = rng.choice(["f32", "bf16"])
    es = 4 if dtype == "f32" else 2
    vocab = _log_int(rng, MIN_VOCAB, CE_VOCAB if kind == "ce" else QWEN_VOCAB)
    if kind == "host":
        return {"kind": kind, "rows": _log_int(rng, 1, 16), "vocab": vocab, **_draw_spread(rng), **_draw_config(rng, vocab)}
    if kind == "sample":
        rows = _log_int(rng, 1, min(1024, MAX_LOGITS_BYTES // (vocab * es)))
        return {"kind": kind, "rows": rows, "vocab": vocab, "dtype": dtype, **_draw_spread(rng), **_draw_config(rng, vocab)}
    if kind == "generate":
        return {"kind": kind, "rows": _log_int(rng, 1, 64), "vocab": vocab, "dtype": dtype, **_draw_spread(rng),
                "new": _log_int(rng, 8, 48), **_draw_config(rng, vocab)}
    if kind in ("lm_sample", "lm_logits"):
        hidden = 64 * _log_int(rng, 8, min(64, MAX_WEIGHTS // (vocab * 64)))
        rows = _log_int(rng, 1, min(512, MAX_LM_MACS // (vocab * hidden)))
        case = {"kind": kind, "rows": rows, "vocab": vocab, "hidden": hidden}
        if kind == "lm_sample":
            case.update(_sampling("rows", round(rng.uniform(0.5, 1.3), 2), _log_int(rng, 5, 100), rng.choice([0.0, 0.9, 0.95]), MODE_B))
        return case
    if kind == "topk":
        return {"kind": kind, "rows": _log_int(rng, 1, 512), "vocab": vocab, "dtype": dtype, "k": _log_int(rng, 1, 1000)}
    if kind == "softmax":
        log, then_draw = rng.choice([False, True]), rng.choice([False, True])
        return {"kind": kind, "rows": _log_int(rng, 1, 512), "vocab": vocab, "dtype": dtype, "log": log,
                "draw": then_draw and not log and dtype == "f32"}
    return {"kind": kind, "rows": _log_int(rng, 16, min(2048, MAX_CE_BYTES // (vocab * 4))), "vocab": vocab, "dtype": dtype}


_handle = None


def _sampler() -> sampling.CudaSampler:
    """The one handle that a program keeps, on PyTorch's stream: its inputs come from there."""
    global _handle
    if _handle is None:
        _handle = sampling.CudaSampler(torch.cuda.current_device())
        _handle.set_stream(torch.cuda.current_stream().cuda_stream)
    return _handle


def _cfgs(case: dict, rows: int) -> np.ndarray:
    cfgs = np.zeros(rows, dtype=CFG_DTYPE)
    for b in range(rows):
        t, k, p = MIXED_CYCLE[b % 4] if case["config"] == "mixed" else (case["temperature"], case["top_k"], case["top_p"])
        cfgs[b] = (t, k, p, case["mode"])
    return cfgs


def _logits(rows: int, vocab: int, dtype: str, sigma: float, peaks: int, peak: float, gen) -> torch.Tensor:
    x = torch.randn(rows, vocab, device="cuda", generator=gen).mul_(sigma)
    if peaks:
        cols = torch.randint(0, vocab, (rows, peaks), device="cuda", generator=gen)
        x.scatter_add_(1, cols, torch.full((rows, peaks), peak, device="cuda"))
    return x.to(TORCH_DTYPES[dtype])


def _ints(n: int) -> torch.Tensor:
    return torch.empty(n, device="cuda", dtype=torch.int32)


class _GivenLogits:
    """The caller's model of a generation, reduced to its answer: logits that lie on the device, other ones for each step."""

    def __init__(self, logits, code: int):
        self.logits, self.code, self.step = logits, code, 0

    def _next(self):
        x = self.logits[self.step % len(self.logits)]
        self.step += 1
        return x.data_ptr(), self.code, x.shape[1], x.shape[1]

    def prefill_dev(self, state):
        self.step = 0
        return self._next()

    def forward_dev(self, state):
        return self._next()


def prepare(case: dict, seed: int) -> dict:
    s = _sampler()
    kind, B, V = case["kind"], case["rows"], case["vocab"]
    st = {"case": case, "s": s}
    if kind == "host":                                    # numpy arrays, as a host-side model hands them over
        rng = np.random.default_rng(seed)
        x = rng.standard_normal((B, V), dtype=np.float32) * np.float32(case["sigma"])
        for b in range(B):
            x[b, rng.integers(0, V, case["peaks"])] += np.float32(case["peak"])
        st.update(x=x, cfgs=_cfgs(case, B), u=rng.random(B))
        return st
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if kind in ("sample", "generate", "lm_sample"):
        cfgs = _cfgs(case, B)
        st.update(cfgs=torch.from_numpy(cfgs.view(np.uint8).reshape(B, 16)).cuda(), ids=_ints(B))
    if kind == "sample":
        st.update(x=_logits(B, V, case["dtype"], case["sigma"], case["peaks"], case["peak"], gen),
                  u=torch.rand(B, device="cuda", dtype=torch.float64, generator=gen))
    elif kind == "generate":
        rng = np.random.default_rng(seed)
        xs = [_logits(B, V, case["dtype"], case["sigma"], case["peaks"], case["peak"], gen) for _ in range(8)]
        st.update(model=_GivenLogits(xs, CODES[case["dtype"]]), host_cfgs=cfgs, u=rng.random((case["new"], B)),
                  prompts=[rng.integers(0, V, 5 + b % 12).tolist() for b in range(B)])
    elif kind in ("lm_sample", "lm_logits"):
        K = case["hidden"]
        st.update(x=(torch.randn(B, K, device="cuda", generator=gen) * 0.5).to(torch.bfloat16),
                  w=(torch.randn(V, K, device="cuda", generator=gen) * (4.0 / math.sqrt(K))).to(torch.bfloat16))
        if kind == "lm_sample":
            st.update(u=torch.rand(B, device="cuda", dtype=torch.float64, generator=gen))
        else:
            st.update(out=torch.empty(B, V, device="cuda"))
    elif kind == "topk":
        k = min(case["k"], V)
        st.update(x=_logits(B, V, case["dtype"], 2.0, 16, 8.0, gen), k=k, values=torch.empty(B, k, device="cuda"),
                  indices=torch.empty(B, k, device="cuda", dtype=torch.int32), flags=_ints(B))
    elif kind == "softmax":
        x = _logits(B, V, case["dtype"], 2.0, 0, 0.0, gen)
        st.update(x=x, out=torch.empty_like(x))
        if case["draw"]:
            st.update(u=torch.rand(B, device="cuda", dtype=torch.float64, generator=gen), ids=_ints(B), flags=_ints(B))
    else:
        st.update(x=_logits(B, V, case["dtype"], 2.0, 0, 0.0, gen),
                  targets=torch.randint(0, V, (B,), device="cuda", dtype=torch.int32, generator=gen),
                  loss=torch.empty(B, device="cuda"), lse=torch.empty(B, device="cuda"), mean=torch.empty(1, device="cuda"),
                  dx=torch.empty(B, V, device="cuda"))
    return st


def _checked(s: sampling.CudaSampler, fn, *args) -> None:
    """A call of the C ABI that has no method of its own on device pointers."""
    err = ctypes.c_void_p()
    rc = fn(s._ctx, *args, ctypes.byref(err))
    sampling._check(s._lib, rc, err)


def run(st: dict):
    case, s = st["case"], st["s"]
    kind, B, V = case["kind"], case["rows"], case["vocab"]
    if kind == "host":
        if B == 1:
            c = st["cfgs"][0]
            return s.sample(st["x"][0], float(c["temperature"]), int(c["top_k"]), float(c["top_p"]), float(st["u"][0]), int(c["topp_mode"]))
        return s.sample_batch(st["x"], st["cfgs"], st["u"], want_flags=False)[0]
    if kind == "sample":
        s.sample_dev_ptrs(st["x"].data_ptr(), CODES[case["dtype"]], B, V, V, st["cfgs"].data_ptr(), st["u"].data_ptr(), st["ids"].data_ptr())
        return st["ids"]
    if kind == "generate":
        out = generate.generate_on_device(st["model"], st["prompts"], st["host_cfgs"], st["u"], s, case["new"], 1 << 20)
        return [np.concatenate([np.asarray(t, dtype=np.int32) for t in out["tokens"]]), out["done"], out["n_new"]]
    if kind == "lm_sample":
        K = case["hidden"]
        s.lm_head_sample_ptrs(st["x"].data_ptr(), K, st["w"].data_ptr(), K, B, V, K, case["top_k"], st["cfgs"].data_ptr(), st["u"].data_ptr(),
                              st["ids"].data_ptr())
        return st["ids"]
    if kind == "lm_logits":
        K = case["hidden"]
        s.lm_head_logits_ptrs(st["x"].data_ptr(), K, st["w"].data_ptr(), K, B, V, K, st["out"].data_ptr(), V)
        return st["out"]
    if kind == "topk":
        _checked(s, s._lib.gorch_cuda_topk_dev, st["x"].data_ptr(), CODES[case["dtype"]], B, V, V, st["k"], st["values"].data_ptr(),
                 st["indices"].data_ptr(), st["flags"].data_ptr())
        return [st["values"], st["indices"], st["flags"]]
    if kind == "softmax":
        row_ops.softmax_ptrs(s, st["x"].data_ptr(), CODES[case["dtype"]], B, V, V, st["out"].data_ptr(), V, case["log"])
        if not case["draw"]:
            return st["out"]
        _checked(s, s._lib.gorch_cuda_multinomial_dev, st["out"].data_ptr(), B, V, V, st["u"].data_ptr(), st["ids"].data_ptr(),
                 st["flags"].data_ptr())
        return [st["out"], st["ids"]]
    x, code, tgt = st["x"].data_ptr(), CODES[case["dtype"]], st["targets"].data_ptr()
    row_ops.cross_entropy_fwd_ptrs(s, x, code, B, V, V, tgt, st["loss"].data_ptr(), st["lse"].data_ptr(), st["mean"].data_ptr())
    row_ops.cross_entropy_bwd_ptrs(s, x, code, B, V, V, tgt, st["lse"].data_ptr(), 1.0 / B, st["dx"].data_ptr(), V)
    return [st["loss"], st["lse"], st["mean"], st["dx"]]


def work(case: dict) -> dict:
    """Each input read once, each output written once. A sampled row: its logits, its 16-byte record, its uniform, its id."""
    kind, B, V = case["kind"], case["rows"], case["vocab"]
    es = 2 if case.get("dtype") == "bf16" else 4
    if kind in ("host", "sample"):
        return {"bytes": B * (V * es + 28), "flops": 0}
    if kind == "generate":
        return {"bytes": case["new"] * B * (V * es + 28), "flops": 0}
    if kind == "lm_sample":
        return {"bytes": (V + B) * case["hidden"] * 2 + B * 28, "flops": 2 * B * V * case["hidden"]}
    if kind == "lm_logits":
        return {"bytes": (V + B) * case["hidden"] * 2 + B * V * 4, "flops": 2 * B * V * case["hidden"]}
    if kind == "topk":
        return {"bytes": B * (V * es + min(case["k"], V) * 8 + 4), "flops": 0}
    if kind == "softmax":
        return {"bytes": B * (2 * V * es + (16 if case["draw"] else 0)), "flops": 4 * B * V}
    return {"bytes": B * (V * es + V * 4 + 12), "flops": 8 * B * V}


def tolerance(case: dict):
    kind = case["kind"]
    if kind == "topk":
        return "exact"
    if kind in ("host", "sample", "generate", "lm_sample"):
        # A uniform that falls within rounding of an edge of its interval may go either way. Where the
        # sums run over the whole vocabulary the intervals are as small as 1e-6, and where logits come out
        # of a bf16 product with f32 sums those carry errors of 1e-6 of their own.
        wide = kind == "lm_sample" or case["config"] == "mixed" or case["top_k"] == 0
        return {"rel": 0.0, "differ": 0.01 if wide else 0.002}
    if kind == "softmax" and case["dtype"] == "bf16":
        return {"rel": 4e-3, "max": 1.6e-2}
    return {"rel": 1e-5, "differ": 0.01}                  # f32 sums; a draw behind a softmax as above
