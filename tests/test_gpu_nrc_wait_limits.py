"""Waits of the network kernels that give up: the kernel reports it, writes no output and no gradient,
waits for what it has started and frees its tensor memory, so that the context and the next calls are as
if it had not run.

A limit of 0 polls makes every wait for a copy, or every wait for a product, give up in all
threads; a few polls may give up in some threads of a warp and not in others."""
import numpy as np
import pytest

from rtc8_gb300 import nrc

from .test_gpu_nrc import _queries, _target

pytestmark = pytest.mark.gpu

CASES = [(nrc.NRC_ENCODING_VOLUME, 5, 20000), (nrc.NRC_ENCODING_VOLUME, 1, 300), (nrc.NRC_ENCODING_REFERENCE, 2, 20000),
         (nrc.NRC_ENCODING_REFERENCE, 7, 1000), (nrc.NRC_ENCODING_HASHGRID, 2, 40000), (nrc.NRC_ENCODING_HASHGRID, 1, 200)]


def _cache(encoding, hidden):
    cfg = nrc.default_config(encoding)
    cfg.num_hidden_layers = hidden
    cfg.ema_decay = 0.0
    cache = nrc.NeuralRadianceCache()
    cache.initialize(config=cfg)
    return cache


@pytest.mark.parametrize("encoding,hidden,n", CASES)
def test_waits_that_give_up(cuda_device, encoding, hidden, n):
    import torch

    q = _queries(n, seed=8, volume=encoding == nrc.NRC_ENCODING_VOLUME)
    qd, td = torch.from_numpy(q).cuda(), torch.from_numpy(np.asarray(_target(q), np.float32)).cuda()
    cache = _cache(encoding, hidden)
    start = cache.params()
    want = torch.zeros((n, 3), device="cuda")
    cache.infer(0, qd, n, want)
    assert cache.device_errors() == 0
    for copy, product in ((0, nrc.WAIT_POLLS), (nrc.WAIT_POLLS, 0), (0, 0)):
        nrc.selftest_wait_limits(cache, copy, product)
        out = torch.full((n, 3), 7.0, device="cuda")
        cache.infer(0, qd, n, out)
        assert cache.device_errors() == 1
        assert bool((out == 7.0).all())
        cache.train(0, qd, td, n)
        assert cache.device_errors() == 1
        assert np.all(cache.gradients() == 0)
        # and straight after it, with the limits as they were
        nrc.selftest_wait_limits(cache)
        cache.set_params(start)
        cache.infer(0, qd, n, out)
        assert cache.device_errors() == 0
        assert torch.equal(out, want)
        assert np.isfinite(cache.train(0, qd, td, n, loss=True))
        assert cache.device_errors() == 0 and np.any(cache.gradients() != 0)
        cache.set_params(start)
    cache.finalize()


@pytest.mark.parametrize("encoding,hidden,n", CASES)
def test_waits_of_a_few_polls(cuda_device, encoding, hidden, n):
    import torch

    q = _queries(n, seed=9, volume=encoding == nrc.NRC_ENCODING_VOLUME)
    qd, td = torch.from_numpy(q).cuda(), torch.from_numpy(np.asarray(_target(q), np.float32)).cuda()
    cache = _cache(encoding, hidden)
    start = cache.params()
    want = torch.zeros((n, 3), device="cuda")
    cache.infer(0, qd, n, want)
    for polls in (1, 2, 3, 5, 8):
        nrc.selftest_wait_limits(cache, nrc.WAIT_POLLS, polls)
        out = torch.full((n, 3), 7.0, device="cuda")
        cache.infer(0, qd, n, out)
        errors = cache.device_errors()
        rows = (out == want).all(dim=1) | (out == 7.0).all(dim=1)   # a row is there or is not
        assert errors in (0, 1) and bool(rows.all()) and (errors or torch.equal(out, want))
        cache.train(0, qd, td, n)
        assert cache.device_errors() in (0, 1)
        assert np.all(np.isfinite(cache.gradients()))
        nrc.selftest_wait_limits(cache)
        cache.set_params(start)
        cache.infer(0, qd, n, out)
        assert cache.device_errors() == 0 and torch.equal(out, want)
    cache.finalize()
