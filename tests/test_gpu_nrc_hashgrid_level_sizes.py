"""Hash-grid inference level by level against the fused kernel at sizes that all reach the level path
(32,768 queries on): networks of one to seven hidden layers at ragged last tiles, and batches of several
chunks whose equal shares end inside a tile. Both do the same arithmetic in the same order: equal to the
bit."""
import pytest

from .test_gpu_nrc_hashgrid import _cache
from .test_gpu_nrc_hashgrid_levels import _inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,hidden", [(32768 + 127, 1), (40001, 2), (50000 - 1, 3), ((1 << 16) + 1, 5), ((1 << 18) + 1, 7),
                                      ((1 << 20) - 1, 1), ((1 << 21) + 1, 2), (3 * (1 << 20) + 129, 4)])
def test_levels_equal_fused(cuda_device, n, hidden):
    import torch

    cache = _cache(hidden=hidden)[0]
    q = _inputs(n, n % 1000)
    a, b = torch.full((n, 3), 7.0, device="cuda"), torch.full((n, 3), 9.0, device="cuda")
    cache.infer(0, q, n, a)
    count = torch.tensor([n], dtype=torch.int32, device="cuda")
    index = torch.arange(n, dtype=torch.int32, device="cuda")
    cache.infer_indexed(0, q, index, count, n, b)   # the fused kernel
    torch.cuda.synchronize()
    assert cache.device_errors() == 0
    assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    cache.finalize()
