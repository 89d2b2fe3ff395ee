"""The narrow kernel's 256-thread instances, with rings of four and of two f32 steps: row lengths at the edges of the warm-up chunk, of a warp's first
steps and of a turn of the ring, unaligned rows, small and large k, greedy rows, ids and kept sets against the oracle."""
import numpy as np
import pytest

from gorch_b200.config import CFG_DTYPE, MODE_A, MODE_B
from tests.test_gpu_parity import run_both

pytestmark = pytest.mark.gpu

WARM, STEP = 4096, 8 * 256                  # logits of the chunk that stays in registers; of a step of all warps


@pytest.mark.parametrize("variant", [2, 7], ids=["four_steps", "two_steps"])
@pytest.mark.parametrize("V", [WARM - 1, WARM + 1, WARM + STEP + 3, WARM + 2 * STEP, WARM + 4 * STEP - 1, WARM + 4 * STEP + 5, WARM + 9 * STEP + 1, 50257])
def test_ring_edges(_sampler_session, oracle, V, variant):
    rng = np.random.Generator(np.random.Philox(key=V))
    cfgs = np.array([(0.8, 40, 0.0, MODE_A), (1.0, 200, 0.95, MODE_B), (0.0, 0, 0.0, MODE_A), (1.3, 1, 0.0, MODE_B), (0.7, 256, 0.6, MODE_A), (1.0, 64, 0.9, MODE_B)],
                    dtype=CFG_DTYPE)
    x = (rng.standard_normal((len(cfgs), V)) * 2).astype(np.float32)
    x[5, :WARM] -= 6.0                       # the chunk lies far below the rest: the hit list fills on the way
    _sampler_session.set_kernel_variant(variant, 0)
    try:
        run_both(_sampler_session, oracle, x, cfgs, rng.random(len(cfgs)), pad=V % 4, allow_tie_cut=True)
    finally:
        _sampler_session.set_kernel_variant(0, 0)
