"""A context that changes its stream while its work is still queued: the calls share scratch memory and the row
lists of the sorted batches, so the later ones have to come behind the earlier ones, and every batch afterwards
has to be whole."""
import numpy as np
import pytest

from gorch_b200.config import CFG_DTYPE, DTYPE_F32, MODE_A, MODE_B
from tests.parity import compare

pytestmark = pytest.mark.gpu

KINDS = [(0.8, 40, 0.0, MODE_A), (1.0, 0, 0.9, MODE_B), (0.0, 0, 0.0, MODE_A), (0.9, 300, 0.0, MODE_A)]   # narrow, wide, greedy, handed over


class _Batch:
    def __init__(self, torch, oracle, B, V, seed):
        rng = np.random.default_rng(seed)
        x = (rng.standard_normal((B, V)) * 2).astype(np.float32)
        self.cfgs = np.zeros(B, dtype=CFG_DTYPE)
        for b in range(B):
            self.cfgs[b] = KINDS[b % len(KINDS)]
        self.u = rng.random(B)
        self.want = oracle.sample_batch(x, self.cfgs, self.u, flags=oracle.FAST_KTH, threads=oracle.hw_threads())
        self.B, self.V = B, V
        self.x, self.du = torch.from_numpy(x).cuda(), torch.from_numpy(self.u).cuda()
        self.dc = torch.from_numpy(self.cfgs.view(np.uint8).reshape(B, 16).copy()).cuda()
        self.out = [(torch.full((B,), -7, dtype=torch.int32, device="cuda"), torch.zeros(B, dtype=torch.int32, device="cuda")) for _ in range(16)]

    def call(self, s, i):
        ids, flags = self.out[i]
        s.sample_dev_ptrs(self.x.data_ptr(), DTYPE_F32, self.B, self.V, self.V, self.dc.data_ptr(), self.du.data_ptr(), ids.data_ptr(), flags.data_ptr())

    def check(self, calls):
        for i in calls:
            got = {"ids": self.out[i][0].cpu().numpy(), "flags": self.out[i][1].cpu().numpy().view(np.uint32)}
            rep = compare(got, self.want, self.u, check_probs=False, allow_tie_cut=True)
            assert rep["id_mismatch"] == rep["boundary_mismatch"]


@pytest.mark.parametrize("B,V", [(400, 6000), (700, 30001)])
def test_batches_across_changes_of_the_stream(_sampler_session, oracle, B, V):
    import torch
    s = _sampler_session
    one, two = _Batch(torch, oracle, B, V, 1), _Batch(torch, oracle, B - 100, V + 1, 2)
    streams = [torch.cuda.Stream().cuda_stream, None, torch.cuda.Stream().cuda_stream, 0]
    s.set_kernel_variant(2, 0)
    torch.cuda.synchronize()
    try:
        for i in range(12):                                  # each call on another stream, none waited for
            s.set_stream(streams[i % len(streams)])
            (one if i % 3 else two).call(s, i)
        s.set_stream(None)
        one.call(s, 12)                                      # and on the last one again
        two.call(s, 13)
        s.sync()
    finally:
        s.set_stream(None)
        s.set_kernel_variant(0, 0)
    torch.cuda.synchronize()
    one.check([i for i in range(12) if i % 3] + [12])
    two.check([i for i in range(12) if not i % 3] + [13])


def test_a_recorded_batch_between_queued_ones(_sampler_session, oracle):
    """The stream that the context goes to is being recorded: the queued work is not drawn into the graph, and the
    stream after it still waits for that work."""
    import torch
    s = _sampler_session
    one = _Batch(torch, oracle, 400, 6000, 3)
    s.set_kernel_variant(2, 0)
    one.call(s, 0)                                           # (grows the context's lists)
    s.sync()
    graph = torch.cuda.CUDAGraph()
    try:
        with torch.cuda.graph(graph, capture_error_mode="thread_local"):
            one.call(s, 1)
            s.set_stream(torch.cuda.current_stream().cuda_stream)
            one.call(s, 2)
            s.set_stream(None)
            one.call(s, 3)
        s.sync()
        one.check([0, 1, 3])
        assert (one.out[2][0].cpu().numpy() == -7).all()
        graph.replay()
        torch.cuda.synchronize()
        one.check([2])
        one.call(s, 4)
        s.sync()
        one.check([4])
    finally:
        s.set_stream(None)
        s.set_kernel_variant(0, 0)
