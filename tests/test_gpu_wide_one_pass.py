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
@pytest.mark.parametrize("V,pad", [(300, 0), (16391, 0), (16403, 1), (20480, 0), (32777, 3), (50257, 2)])
def test_one_pass_rows(wide, oracle, V, pad, bf16):
    x, cfgs, one, u = _batch(V, 7000 + V)
    if bf16:
        x = oracle.f32_to_bf16_bits(x)
    gpu, _, _ = run_both(wide, oracle, x, cfgs, u, pad=pad, allow_tie_cut=True)
    paths = gpu["debug"]["path"]
    assert np.all(paths[one & (cfgs["top_p"] == 0.0)] == 3)             # no cut: always one pass
    if V == 50257 and not bf16:
        assert paths[0] == 3 and paths[1] == 3                        # flat rows under a deep nucleus


# reserved[6] of a wide row's debug record: why it took two passes
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


def test_uniforms_at_the_ends(wide, oracle):
    """u = 0 takes the first kept logit, the largest u below 1 the last one."""
    rng = np.random.Generator(np.random.Philox(key=31))
    V = 40000
    x = np.repeat((rng.standard_normal((1, V)) * 0.25).astype(np.float32), 6, axis=0)
    cfgs = np.array([(1.0, 0, 0.99, MODE_B), (1.0, 0, 0.0, MODE_B)] * 3, dtype=CFG_DTYPE)
    u = np.array([0.0, 0.0, np.nextafter(1.0, 0.0), np.nextafter(1.0, 0.0), 0.5, 0.5])
    run_both(wide, oracle, x, cfgs, u)
