"""Training steps whose kernels start while their predecessors drain: steps queued back to back,
steps with a wait after each, and steps replayed from a captured CUDA graph give the same weights up
to the order of the gradient's atomic additions; the gradient the caller reads is the last step's,
and a step of few or ragged records leaves nothing behind for the next one.

Tolerance: the atomics change a gradient by a few FP32 roundings (2^-24 each, over at most 128
addends: 1e-5 relative); Adam's normalised step passes that on to a weight as at most the learning
rate times the relative change, except where a gradient is itself only rounding noise, so the
weights are compared as vectors (relative L2 1e-3 after four steps at lr 1e-3)."""
import numpy as np
import pytest

from rtc8_gb300 import nrc

from .test_gpu_nrc import _queries, _target

pytestmark = pytest.mark.gpu

CASES = [(nrc.NRC_ENCODING_VOLUME, 5, 16384), (nrc.NRC_ENCODING_VOLUME, 1, 129), (nrc.NRC_ENCODING_REFERENCE, 2, 1000),
         (nrc.NRC_ENCODING_REFERENCE, 7, 20000), (nrc.NRC_ENCODING_HASHGRID, 2, 16384), (nrc.NRC_ENCODING_HASHGRID, 1, 300)]


def _cache(encoding, hidden):
    cfg = nrc.default_config(encoding)
    cfg.num_hidden_layers = hidden
    cfg.learning_rate = 1e-3
    cache = nrc.NeuralRadianceCache()
    cache.initialize(config=cfg)
    return cache


def _close(a, b):
    assert np.linalg.norm(a - b) <= 1e-3 * np.linalg.norm(b)


@pytest.mark.parametrize("encoding,hidden,n", CASES)
def test_queued_steps_equal_separate_steps(cuda_device, encoding, hidden, n):
    import torch

    q = _queries(n, seed=5, volume=encoding == nrc.NRC_ENCODING_VOLUME)
    qd, td = torch.from_numpy(q).cuda(), torch.from_numpy(np.asarray(_target(q), np.float32)).cuda()
    a, b = _cache(encoding, hidden), _cache(encoding, hidden)
    for _ in range(4):
        a.train(0, qd, td, n)
    losses = []
    for _ in range(4):
        losses.append(b.train(0, qd, td, n, loss=True))
        torch.cuda.synchronize()
    _close(a.params(), b.params())
    assert np.all(np.isfinite(losses)) and losses[3] < losses[0]
    ga, gb = a.gradients(), b.gradients()
    assert np.linalg.norm(ga - gb) <= 2e-2 * np.linalg.norm(gb) and np.linalg.norm(gb) > 0
    # One record afterwards: its gradient is its own, nothing of the steps before is left in it.
    c = _cache(encoding, hidden)
    c.set_params(a.params())
    a.train(0, qd, td, 1)
    c.train(0, qd, td, 1)
    np.testing.assert_allclose(a.gradients(), c.gradients(), rtol=1e-4, atol=1e-6 * np.abs(c.gradients()).max())
    assert a.device_errors() == b.device_errors() == c.device_errors() == 0
    for x in (a, b, c):
        x.finalize()


@pytest.mark.parametrize("encoding,hidden,n", [CASES[0], CASES[4]])
def test_captured_step_replays(cuda_device, encoding, hidden, n):
    """A captured step replays with the bias corrections it was captured with (its second step)."""
    import torch

    q = _queries(n, seed=6, volume=encoding == nrc.NRC_ENCODING_VOLUME)
    qd, td = torch.from_numpy(q).cuda(), torch.from_numpy(np.asarray(_target(q), np.float32)).cuda()
    a, b = _cache(encoding, hidden), _cache(encoding, hidden)
    a.train(0, qd, td, n)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        a.train(torch.cuda.current_stream().cuda_stream, qd, td, n)
    g.replay()
    torch.cuda.synchronize()
    for _ in range(2):
        b.train(0, qd, td, n)
    _close(a.params(), b.params())
    grad = a.gradients()
    g.replay()
    torch.cuda.synchronize()
    assert np.linalg.norm(a.gradients()) < 1.5 * np.linalg.norm(grad)  # one step's, not a sum of several
    assert a.device_errors() == 0
    a.finalize()
    b.finalize()
