"""Launches of several contexts at once give the images they give alone: contexts of different launch
shapes, grids and majorant modes, each on its own thread and stream, render, start over and read their
own image while the others are launching; the same from one thread that launches them in turn.

Configuration streams add a pixel's samples with FP64 atomics in launch order (sums to 1e-12); RNG
states and decision logs are equal to the bit."""
import threading

import numpy as np
import pytest

from rtc8_gb300.renderer import Renderer, constant_environment, setup_scene

from ._scenes import small_config_mode, small_reference_mode, volume_for

pytestmark = pytest.mark.gpu

SPP = 2
JOBS = [(small_config_mode(size=24, n=24), 0), (small_config_mode(size=40, n=40), 32), (small_reference_mode(size=32, n=24), 96),
        (small_config_mode(size=56, n=40), 128), (small_reference_mode(size=24, n=40), 64), (small_config_mode(size=33, n=17), 0)]


def _context(cfg, threads):
    r = Renderer(cfg.width, cfg.height)
    setup_scene(r, cfg, volume=volume_for(cfg))
    r.set_environment_rgb(constant_environment(cfg.env_constant if cfg.env_constant is not None else 0.5))
    r.set_launch_shape(0, threads, 0)
    return r


def _render(r, cfg, stream, log):
    """The image of a fresh sequence: RNG, accumulation and streams start over (set-up calls run on the
    default stream, so the context's own launches are waited for first)."""
    stream.synchronize()
    r.seed_rng(cfg.rng_seed)
    r.launch_plain_logged(SPP, log.data_ptr(), stream.cuda_stream)
    stream.synchronize()
    return log.cpu().numpy(), r.rng_states(), r.download_sum()[0], r.download_mean()


def _buffers(cfg):
    import torch

    return torch.cuda.Stream(), torch.zeros(cfg.width * cfg.height * SPP * 4, dtype=torch.int32, device="cuda")


def _alone():
    out = []
    for cfg, threads in JOBS:
        r = _context(cfg, threads)
        out.append(_render(r, cfg, *_buffers(cfg)))
        r.close()
    return out


def _check(got, want):
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])
    np.testing.assert_allclose(got[2], want[2], rtol=1e-12, atol=1e-15)
    np.testing.assert_allclose(got[3], want[3], rtol=1e-6, atol=1e-9)


def test_threads_render_their_own_images(cuda_device):
    import torch

    want = _alone()
    bufs = [_buffers(cfg) for cfg, _ in JOBS]
    torch.cuda.synchronize()
    start = threading.Barrier(len(JOBS))
    failed = []

    def work(k):
        try:
            cfg, shape = JOBS[k]
            r = _context(cfg, shape)
            start.wait(60)
            for _ in range(12):
                for _ in range(5):
                    r.launch_plain(SPP, bufs[k][0].cuda_stream)
                _check(_render(r, cfg, *bufs[k]), want[k])
            assert r.device_errors() == 0
            r.close()
        except Exception as e:  # the thread's failure is reported by the test
            failed.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(JOBS))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed


def test_streams_of_one_thread_render_their_own_images(cuda_device):
    import torch

    want = _alone()
    bufs = [_buffers(cfg) for cfg, _ in JOBS]
    rs = [_context(cfg, threads) for cfg, threads in JOBS]
    torch.cuda.synchronize()
    for _ in range(3):
        for r, (cfg, _), (s, log) in zip(rs, JOBS, bufs):
            r.launch_plain(3, s.cuda_stream)
            s.synchronize()
            r.seed_rng(cfg.rng_seed)
        for r, (s, log) in zip(rs, bufs):
            r.launch_plain_logged(SPP, log.data_ptr(), s.cuda_stream)
        torch.cuda.synchronize()
        for r, (s, log), w in zip(rs, bufs, want):
            _check((log.cpu().numpy(), r.rng_states(), r.download_sum()[0], r.download_mean()), w)
            assert r.device_errors() == 0
    for r in rs:
        r.close()
