"""Large hash-grid inference batches compute the grid features level by level through a workspace;
small batches, batches with a device-side count and batches under stream capture gather them inside
the MLP kernel. Both do the same arithmetic in the same order: equal to the bit, at the threshold,
at ragged tiles, over a chunk boundary, for positions on lattice points, outside the box and NaN,
and when several streams infer with one cache at once."""
import numpy as np
import pytest

from .test_gpu_nrc import _queries
from .test_gpu_nrc_hashgrid import _cache

pytestmark = pytest.mark.gpu


def _inputs(n, seed):
    import torch

    q = np.asarray(_queries(1024, seed=seed), dtype=np.float32)
    q = np.tile(q, (n // 1024 + 1, 1))[:n].copy()
    rng = np.random.default_rng(seed)
    q[:, :3] = rng.random((n, 3), dtype=np.float32)
    q[::97, :3] = rng.integers(0, 17, (len(q[::97]), 3)) / np.float32(16)
    q[5::131, 0] = -0.25
    q[7::131, 1] = 1.75
    q[11::4099, 2] = np.nan
    return torch.from_numpy(q).cuda()


@pytest.mark.parametrize("n,hidden", [(16383, 2), (16384, 2), (16385, 1), (20001, 7), (32767, 2), (32768, 1), (32769, 7),
                                      ((1 << 20) + 77, 2)])
def test_levels_equal_fused(cuda_device, n, hidden):
    import torch

    cache = _cache(hidden=hidden)[0]
    q = _inputs(n, 3)
    a, b = torch.full((n, 3), 7.0, device="cuda"), torch.full((n, 3), 9.0, device="cuda")
    cache.infer(0, q, n, a)
    count = torch.tensor([n], dtype=torch.int32, device="cuda")
    index = torch.arange(n, dtype=torch.int32, device="cuda")
    cache.infer_indexed(0, q, index, count, n, b)   # the fused kernel
    torch.cuda.synchronize()
    assert cache.device_errors() == 0
    assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    cache.finalize()


def test_streams_and_capture(cuda_device):
    import torch

    cache = _cache()[0]
    n = 40000
    qs = [_inputs(n, k) for k in range(4)]
    want = [torch.empty((n, 3), device="cuda") for _ in qs]
    for q, w in zip(qs, want):
        cache.infer(0, q, n, w)
    torch.cuda.synchronize()
    outs = [torch.zeros((n, 3), device="cuda") for _ in qs]
    streams = [torch.cuda.Stream() for _ in qs]
    for _ in range(3):
        for s, q, o in zip(streams, qs, outs):
            cache.infer(s.cuda_stream, q, n, o)
    torch.cuda.synchronize()
    captured = torch.zeros((n, 3), device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        cache.infer(torch.cuda.current_stream().cuda_stream, qs[0], n, captured)
    g.replay()
    torch.cuda.synchronize()
    for o, w in zip(outs + [captured], want + [want[0]]):
        assert torch.equal(o.view(torch.int32), w.view(torch.int32))
    assert cache.device_errors() == 0
    cache.finalize()
