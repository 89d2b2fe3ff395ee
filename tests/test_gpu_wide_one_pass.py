"""Rows without top-k in one pass: lengths at the edges of the sample, of a step and of a piece, unaligned rows, windows in the middle
of the logits and down to their end, cuts inside runs of equal logits (also runs longer than the selection's candidates), an anchor that
has to rise, masked logits. Both instances of the wide kernel, through the C ABI against the oracle with the usual gates."""
import numpy as np
import pytest

from gorch_b200.config import CFG_DTYPE, MODE_A, MODE_B
from tests.test_gpu_parity import run_both

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[4, 5], ids=["w256", "w1024"])
def wide(request, _sampler_session):
    _sampler_session.set_kernel_variant(request.param, 0)
    _sampler_session.variant = request.param
    _sampler_session.one_pass_from = {4: 32832, 5: 65600}[request.param]   # shorter rows with a cut are not sampled
    yield _sampler_session
    _sampler_session.set_kernel_variant(0, 0)


def _batch(V, seed):
    """Rows, their configurations and which of them must be served by one pass (w256)."""
    rng = np.random.Generator(np.random.Philox(key=seed))
    rows, cfgs, one = [], [], []

    def add(x, T, p, mode, single):
        rows.append(x.astype(np.float32)); cfgs.append((T, 0, p, mode)); one.append(single)

    z = lambda s: rng.standard_normal(V) * s
    add(z(0.25), 1.0, 0.99, MODE_B, False)
    add(z(0.25), 0.83, 0.995, MODE_B, False)
    add(z(0.1) - 3.0, 1.0, 0.97, MODE_B, False)
    add(np.round(z(0.25) * 512) / 512, 1.0, 0.99, MODE_B, False)      # runs of a few equal logits at the cut
    add(np.round(z(0.25) * 16) / 16, 1.1, 0.99, MODE_B, False)        # runs of hundreds
    add(np.round(z(0.25) * 16) / 16, 1.0, 0.64, MODE_A, False)        # ... of which mode A drops the lowest indices first
    add(z(0.25), 1.0, 0.65, MODE_A, False)
    add(z(2.0), 1.0, 0.0, MODE_B, True)
    x = z(2.0); x[V // 3] += 25.0; x[V - 1] += 40.0                    # the anchor rises twice
    add(x, 0.9, 0.0, MODE_A, True)
    add(np.sort(z(3.0)), 1.0, 0.0, MODE_A, True)                      # ... and in every warp
    x = z(0.25); x[rng.random(V) < 0.3] = -np.inf
    add(x, 1.0, 0.99, MODE_B, False)
    x = z(1.0); x[5:] = -np.inf
    add(x, 1.0, 0.0, MODE_B, False)
    x = z(0.25); x[V // 2] = 30.0                                      # all mass on one logit that no sample holds
    add(x, 1.0, 0.99, MODE_B, False)
    return np.stack(rows), np.array(cfgs, dtype=CFG_DTYPE), np.array(one), rng.random(len(rows))


@pytest.mark.parametrize("bf16", [False, True], ids=["f32", "bf16"])
@pytest.mark.parametrize("V,pad", [(300, 0), (16391, 0), (16403, 1), (20480, 0), (32777, 3), (50257, 2), (70001, 1)])
def test_one_pass_rows(wide, oracle, V, pad, bf16):
    x, cfgs, one, u = _batch(V, 7000 + V)
    if bf16:
        x = oracle.f32_to_bf16_bits(x)
    gpu, _, _ = run_both(wide, oracle, x, cfgs, u, pad=pad, allow_tie_cut=True)
    paths = gpu["debug"]["path"]
    assert np.all(paths[one & (cfgs["top_p"] == 0.0)] == 3)             # no cut: always one pass
    if V >= 50257:                                                      # flat rows under a deep nucleus, with short runs and with masked logits too
        assert np.all(paths[[0, 1, 3, 6, 10]] == (2 if wide.one_pass_from > V else 3))
        assert paths[12] == 2                                           # (the maximum far above the sample's)


# Normal rows, their top-p, the passes they take, and by which means: the lanes' buffers emptied more often, or twice the sample. What a row's window holds is
# known to a tenth, so every case lies that far from a line.
REACH = {4: [(33000, 0.25, 0.9, 3, "often"), (50257, 0.25, 0.7, 2, ""), (50257, 0.25, 0.93, 3, "often"), (50257, 0.25, 0.99, 3, ""), (100003, 0.25, 0.9, 2, ""),
             (100003, 0.25, 0.97, 3, "often"), (151936, 0.25, 0.9, 2, ""), (151936, 0.25, 0.98, 3, "twice"), (151936, 0.4, 0.99, 3, "twice"), (151936, 0.25, 0.99, 3, "")],
         5: [(70001, 0.25, 0.7, 2, ""), (100003, 0.25, 0.97, 3, "often"), (151936, 0.25, 0.9, 2, ""), (151936, 0.25, 0.98, 3, "")]}
HOW_CUT, HOW_LOW, HOW_ONE_CLASS, HOW_BY_PIECE, HOW_INDEX, HOW_EXACT, HOW_OFTEN, HOW_TWICE = (1 << i for i in range(8))


@pytest.mark.parametrize("bf16", [False, True], ids=["f32", "bf16"])
def test_reach_of_rows_with_a_cut(wide, oracle, bf16):
    """Rows on both sides of the lines: the lanes' buffers emptied more often, the other half of the sample, windows too wide for the lists."""
    rng = np.random.Generator(np.random.Philox(key=501))
    for V, sigma, p, path, extra in REACH[wide.variant]:
        x = (rng.standard_normal((4, V)) * sigma).astype(np.float32)
        cfgs = np.array([(1.0, 0, p, MODE_B)] * 3 + [(1.25, 0, p / 1.5, MODE_A)], dtype=CFG_DTYPE)
        x[3] *= np.float32(1.25)
        gpu, _, _ = run_both(wide, oracle, oracle.f32_to_bf16_bits(x) if bf16 else x, cfgs, rng.random(4), pad=V % 4, allow_tie_cut=True, want_probs=False)
        d = gpu["debug"]
        assert list(d["path"]) == [path] * 4, (V, sigma, p)
        how = d["reserved"][:, 7]
        assert np.all(((how & HOW_OFTEN) != 0) == (extra == "often")) and np.all(((how & HOW_TWICE) != 0) == (extra == "twice")), (V, sigma, p)
        if path == 2:
            assert np.all(d["reserved"][:, 6] == WHY_WINDOW)


@pytest.mark.parametrize("bf16", [False, True], ids=["f32", "bf16"])
def test_cut_inside_runs(wide, oracle, bf16):
    """The cut divides runs of 2 to 32 equal logits (steps of 1/1,024, f32), which the selection looks at one by one, and runs of hundreds (1/64), in
    both modes: all of it in one pass, the member's index from a piece that is read again."""
    rng = np.random.Generator(np.random.Philox(key=502))
    V = {4: 50257, 5: 66001}[wide.variant]
    rows, cfgs = [], []
    for q in (1024, 64):
        for p, mode in ((0.99, MODE_B), (0.987, MODE_B), (0.985, MODE_B), (0.66, MODE_A), (0.658, MODE_A), (0.6565, MODE_A)):
            rows.append(np.round(rng.standard_normal(V) * 0.25 * q) / q)
            cfgs.append((1.0, 0, p, mode))
    x = np.stack(rows).astype(np.float32)
    gpu, _, _ = run_both(wide, oracle, oracle.f32_to_bf16_bits(x) if bf16 else x, np.array(cfgs, dtype=CFG_DTYPE), rng.random(len(rows)), allow_tie_cut=True)
    how = gpu["debug"]["reserved"][:, 7]
    assert np.all(gpu["debug"]["path"] == 3)
    for b in (0, 3, 6, 9):                                   # (a cut may fall on the end of a run)
        assert np.sum((how[b:b + 3] & (HOW_BY_PIECE | HOW_INDEX)) == (HOW_BY_PIECE | HOW_INDEX)) >= 2
    assert np.all(how[6:] & HOW_ONE_CLASS) and (bf16 or not np.any(how[:6] & HOW_ONE_CLASS))


# reserved[6] of a wide row's debug record: why it took two passes; reserved[7]: what one pass did
WHY_TEMPERATURE, WHY_SHORT, WHY_NOT_FINITE, WHY_HEAVY, WHY_WINDOW, WHY_EMPTY_WINDOW, WHY_NAN, WHY_LIST, WHY_ANCHOR = range(1, 10)


def test_reasons_for_two_passes(wide, oracle):
    """The record says why a row was not served by one pass."""
    rng = np.random.Generator(np.random.Philox(key=77))
    V = 70000
    z = lambda s: (rng.standard_normal(V) * s).astype(np.float32)
    rows, cfgs, why = [], [], []
    for x, T, p, w in ((z(0.25), 1.0, 0.995, 0), (z(2.0), 1.0, 0.0, 0), (z(0.25), 1.0, 0.5, WHY_WINDOW), (z(2.5), 1.0, 0.9, WHY_HEAVY),
                       (z(0.25), np.nextafter(np.float32(2.0), np.float32(0.0)), 0.0, WHY_TEMPERATURE)):
        rows.append(x); cfgs.append((T, 0, p, MODE_B)); why.append(w)
    x = z(2.0); x[V // 2] = np.nan
    rows.append(x); cfgs.append((1.0, 0, 0.0, MODE_B)); why.append(WHY_NAN)
    x = z(0.25); x[:] = -np.inf
    rows.append(x); cfgs.append((1.0, 0, 0.9, MODE_B)); why.append(WHY_NOT_FINITE)
    gpu, _, _ = run_both(wide, oracle, np.stack(rows), np.array(cfgs, dtype=CFG_DTYPE), rng.random(len(rows)))
    assert list(gpu["debug"]["reserved"][:, 6]) == why
    assert list(gpu["debug"]["path"]) == [2 if w else 3 for w in why]


@pytest.mark.parametrize("bf16", [False, True], ids=["f32", "bf16"])
@pytest.mark.parametrize("V", [300, 16391, 70001])
def test_sums_without_a_cut(wide, oracle, V, bf16):
    """The softmax denominator of rows without a cut against the sum in 64 bits, wherever the row lies. An exact exponential is off by
    1.2e-10 + 2.4e-12 per unit below the maximum (of 30 that matter), and so is a sum of them; 1e-12 for 1e5 additions in f64."""
    rng = np.random.Generator(np.random.Philox(key=91 + V))
    z = lambda s: rng.standard_normal(V) * s
    rows, T = [], []
    for x, t in ((z(2.0), 1.0), (z(0.25), 0.8), (z(3.0) + 1000.0, 1.0), (z(3.0) - 1000.0, 1.3), (z(2.0), 0.07), (z(2.0) + 31.0, 1.0), (z(2.0) - 33.0, 1.0),
                 (z(1.0) + 5e5, 1.0)):
        rows.append(x); T.append(t)
    x = z(1.0); x[V - 1] = 70.0                              # all but one token far below a maximum that the first look misses
    rows.append(x); T.append(1.0)
    x = z(2.0); x[: V // 2] = -np.inf
    rows.append(x); T.append(0.7)
    x = np.stack(rows).astype(np.float32)
    cfgs = np.array([(t, 0, 0.0, MODE_B) for t in T], dtype=CFG_DTYPE)
    bits = oracle.f32_to_bf16_bits(x) if bf16 else x
    if bf16:
        x = (bits.astype(np.uint32) << 16).view(np.float32)
    gpu, _, _ = run_both(wide, oracle, bits, cfgs, rng.random(len(T)))
    assert np.all(gpu["debug"]["path"] == 3)
    exact = (gpu["debug"]["reserved"][:, 7] & HOW_EXACT) != 0
    assert np.all(exact[[0, 2, 3, 4, 5, 6, 8]]) and (V > 16000 or np.all(exact))
    s = (x / np.array(T, dtype=np.float32)[:, None]).astype(np.float64)
    want = np.exp(s - s.max(axis=1, keepdims=True)).sum(axis=1)
    err = np.abs(gpu["debug"]["sum_exp"] / want - 1.0)
    assert np.max(err[exact]) <= 1.2e-10 + 30 * 2.4e-12 + 1e-12
    assert np.all(err <= 4.5e-7 + 2.0e-7 * 9.7)             # the budget of the quick sums


def test_maxima_far_from_the_first_look(wide, oracle):
    """Short rows (and those whose first look spans much) take the exact sums at once, and a maximum more than 88 above their base leaves them to the two-pass form; a long
    row's quick sums end at the first logit that is too far up, and the exact ones know it. Beyond 1e6 there are no exact sums."""
    rng = np.random.Generator(np.random.Philox(key=5))
    cfgs = np.array([(1.0, 0, 0.0, MODE_A)] * 5, dtype=CFG_DTYPE)
    for V, path, why in ((10000, [3, 2, 2, 2, 3], [0, WHY_ANCHOR, WHY_ANCHOR, WHY_ANCHOR, 0]),
                         (70000, [3] * 5, [0] * 5)):
        x = (rng.standard_normal((5, V)) * 0.25).astype(np.float32)
        x[0, V - 1] = 87.0; x[1, V - 1] = 89.0; x[2] += 2e6; x[3] -= 2e6
        gpu, _, _ = run_both(wide, oracle, x, cfgs, rng.random(5))
        assert list(gpu["debug"]["path"]) == path and list(gpu["debug"]["reserved"][:, 6]) == why
        how = gpu["debug"]["reserved"][:, 7] & HOW_EXACT
        assert list(how != 0) == ([True, False, False, False, True] if V == 10000 else [True, True, False, False, False])


@pytest.mark.parametrize("bf16", [False, True], ids=["f32", "bf16"])
def test_shortest_row_with_a_cut_in_one_pass(wide, oracle, bf16):
    rng = np.random.Generator(np.random.Philox(key=12))
    for V, pad, path, why in ((wide.one_pass_from - 1, 1, 2, WHY_SHORT), (wide.one_pass_from, 0, 3, 0), (wide.one_pass_from + 5, 3, 3, 0)):
        x = (rng.standard_normal((6, V)) * 0.25).astype(np.float32)
        cfgs = np.array([(T, 0, p, MODE_B) for T in (1.0, 0.8) for p in (0.99, 0.995, 0.999)], dtype=CFG_DTYPE)
        gpu, _, _ = run_both(wide, oracle, oracle.f32_to_bf16_bits(x) if bf16 else x, cfgs, rng.random(6), pad=pad, allow_tie_cut=True)
        assert np.all(gpu["debug"]["path"] == path) and np.all(gpu["debug"]["reserved"][:, 6] == why)


@pytest.mark.parametrize("T", [1.0, 0.8])
def test_cut_at_the_end_of_a_run(wide, oracle, T):
    """Long runs of equal logits, and a top-p within a few ulps of the mass through one of them: the bounds that look for the
    cut's run cannot tell it from the next, and one pass has to find it all the same."""
    rng = np.random.Generator(np.random.Philox(key=41))
    V = 90000
    base = (np.round(rng.standard_normal(V) * 0.25 * 64) / 64).astype(np.float32)
    s = base / np.float32(T)
    e = np.exp((s - s.max()).astype(np.float64))
    vals, n = np.unique(s, return_counts=True)
    through = np.cumsum((np.exp((vals - vals.max()).astype(np.float64)) * n)[::-1]) / e.sum()
    cuts = through[np.flatnonzero((through > 0.988) & (through < 0.997) & (n[::-1] > 40))][:6]
    assert len(cuts) >= 4
    ps = [np.float32(c) + np.float32(k * 2.0 ** -24) for c in cuts for k in (-2, 0, 2)]
    x = np.repeat(base[None], len(ps), axis=0)
    cfgs = np.array([(T, 0, p, MODE_B) for p in ps], dtype=CFG_DTYPE)
    gpu, _, _ = run_both(wide, oracle, x, cfgs, rng.random(len(ps)), allow_tie_cut=True)
    assert list(gpu["debug"]["reserved"][:, 6]) == [0] * len(ps) and np.all(gpu["debug"]["path"] == 3)


def test_uniforms_at_the_ends(wide, oracle):
    """u = 0 takes the first kept logit, the largest u below 1 the last one."""
    rng = np.random.Generator(np.random.Philox(key=31))
    V = 70000
    x = np.repeat((rng.standard_normal((1, V)) * 0.25).astype(np.float32), 6, axis=0)
    cfgs = np.array([(1.0, 0, 0.99, MODE_B), (1.0, 0, 0.0, MODE_B)] * 3, dtype=CFG_DTYPE)
    u = np.array([0.0, 0.0, np.nextafter(1.0, 0.0), np.nextafter(1.0, 0.0), 0.5, 0.5])
    gpu, _, _ = run_both(wide, oracle, x, cfgs, u)
    assert np.all(gpu["debug"]["path"] == 3)


def test_finite_logits_far_out(wide, oracle):
    """A finite maximum of 1e32, outside what a first look sees, without a cut: no base serves the row, and two passes take that very token."""
    rng = np.random.Generator(np.random.Philox(key=33))
    for V in (10000, 70000):
        x = (rng.standard_normal((2, V)) * 0.25).astype(np.float32)
        x[:, V // 2 + 100] = 1e32
        gpu, _, _ = run_both(wide, oracle, x, np.array([(1.0, 0, 0.0, MODE_A), (0.9, 0, 0.0, MODE_B)], dtype=CFG_DTYPE), rng.random(2))
        assert np.all(gpu["ids"] == V // 2 + 100)
        assert np.all(gpu["debug"]["path"] == 2) and np.all(gpu["debug"]["reserved"][:, 6] == WHY_ANCHOR)


def test_limit_between_two_threads(wide, oracle):
    """Rows whose window's limit falls into the rounding between one thread's prefix of the sample's mass and the next one's."""
    V, keys = {4: (50257, (9803, 11332)), 5: (70001, (2272, 5846))}[wide.variant]
    x = np.stack([np.random.Generator(np.random.Philox(key=k)).standard_normal(V, dtype=np.float32) * np.float32(0.25) for k in keys])
    gpu, _, _ = run_both(wide, oracle, x, np.array([(1.0, 0, 0.99, MODE_B)] * len(keys), dtype=CFG_DTYPE), np.full(len(keys), 0.5))
    assert list(gpu["debug"]["reserved"][:, 6]) == [0] * len(keys) and np.all(gpu["debug"]["path"] == 3)
