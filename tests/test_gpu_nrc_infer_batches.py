"""Inference spreads the 128-row tiles of a batch over the SMs in turn, and the groups of a CTA wait
for one copy of the weights. A query's result depends on neither: batches of every shape (one row, tile
edges, fewer tiles than SMs, around one and four tiles per SM, device-side counts of none and of a part
of the batch) equal the same rows of a large batch to the bit, which other tests compare with the
oracle."""
import numpy as np
import pytest

from rtc8_gb300 import nrc

from .test_gpu_nrc import _queries

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("encoding,hidden", [(nrc.NRC_ENCODING_VOLUME, 5), (nrc.NRC_ENCODING_VOLUME, 1),
                                             (nrc.NRC_ENCODING_REFERENCE, 2), (nrc.NRC_ENCODING_REFERENCE, 7)])
def test_batch_shapes(cuda_device, encoding, hidden):
    import torch

    cfg = nrc.default_config(encoding)
    cfg.num_hidden_layers = hidden
    cache = nrc.NeuralRadianceCache()
    cache.initialize(config=cfg)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    most = 128 * 9 * sms + 5
    rows = _queries(1024, 3, volume=encoding == nrc.NRC_ENCODING_VOLUME)
    q = torch.from_numpy(np.tile(rows, (most // 1024 + 1, 1))[:most].copy()).cuda()
    q[:, :3] = torch.rand((most, 3), device="cuda", generator=torch.Generator("cuda").manual_seed(5))
    full = torch.zeros((most, 3), device="cuda")
    cache.infer(0, q, most, full)
    for n in (1, 127, 128, 129, 1000, 128 * sms - 1, 128 * sms + 1, 128 * 4 * sms, 128 * 4 * sms + 1):
        out = torch.full((most, 3), -7.0, device="cuda")
        cache.infer(0, q, n, out)
        assert torch.equal(out[:n], full[:n]) and bool((out[n:] == -7.0).all())
    index = torch.arange(most, dtype=torch.int32, device="cuda")
    for n in (0, 1, 129, 128 * sms + 1):
        out = torch.full((most, 3), -7.0, device="cuda")
        cache.infer_indexed(0, q, index, torch.tensor([n], dtype=torch.int32, device="cuda"), most, out)
        assert torch.equal(out[:n], full[:n]) and bool((out[n:] == -7.0).all())
    torch.cuda.synchronize()
    assert cache.device_errors() == 0
    cache.finalize()


@pytest.mark.parametrize("encoding,deep", [(nrc.NRC_ENCODING_VOLUME, 5), (nrc.NRC_ENCODING_REFERENCE, 7),
                                           (nrc.NRC_ENCODING_HASHGRID, 7)])
def test_caches_of_different_depths(cuda_device, encoding, deep):
    """A deep network's cache still infers and trains after a shallow one was created (they share the
    kernels), and gives the same outputs as before."""
    import torch

    def cache(hidden):
        cfg = nrc.default_config(encoding)
        cfg.num_hidden_layers = hidden
        c = nrc.NeuralRadianceCache()
        c.initialize(config=cfg)
        return c

    n = 3000
    q = torch.from_numpy(_queries(n, 3, volume=encoding == nrc.NRC_ENCODING_VOLUME)).cuda()
    a, b, t = torch.zeros((n, 3), device="cuda"), torch.ones((n, 3), device="cuda"), torch.full((n, 3), 0.5, device="cuda")
    first = cache(deep)
    first.infer(0, q, n, a)
    second = cache(1)
    second.infer(0, q, n, b)
    first.infer(0, q, n, b)
    torch.cuda.synchronize()
    assert torch.equal(a, b)
    before = first.params().copy()
    first.train(0, q, t, n)
    second.train(0, q, t, n)
    assert np.isfinite(first.params()).all() and (first.params() != before).any()
    assert first.device_errors() == 0 and second.device_errors() == 0
    first.finalize()
    second.finalize()
