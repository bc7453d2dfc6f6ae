"""The tracker with work queues at the sizes where its queues can go wrong: fewer items than slots,
one item, images that are no multiple of anything, CTAs of one warp up to the default, and launches
that refill every slot many times. The wavefront tracker draws every path's random numbers in the same order,
so decision logs, RNG states and means are equal to the bit."""
import numpy as np
import pytest

from rtc8_gb300.renderer import Renderer, constant_environment, setup_scene

from ._scenes import small_config_mode, small_reference_mode, volume_for

pytestmark = pytest.mark.gpu


def _render(cfg, vox, spp, tracker, threads=0, ctas=0):
    import torch

    r = Renderer(cfg.width, cfg.height)
    setup_scene(r, cfg, volume=vox)
    r.set_environment_rgb(constant_environment(cfg.env_constant if cfg.env_constant is not None else 0.5))
    r.set_tracker(tracker)
    r.set_launch_shape(ctas, threads, 0)
    log = torch.zeros(cfg.width * cfg.height * spp * 4, dtype=torch.int32, device="cuda")
    r.launch_plain_logged(spp, log.data_ptr())
    r.synchronize()
    out = (log.cpu().numpy(), r.rng_states(), r.download_mean(), r.download_sum()[0], r.counters(), r.device_errors())
    r.close()
    return out


@pytest.mark.parametrize("mode", ["reference", "config"])
@pytest.mark.parametrize("width,height,spp,threads,ctas", [(1, 1, 1, 0, 0), (1, 1, 9, 32, 1), (3, 2, 5, 32, 0),
                                                          (33, 17, 7, 96, 0), (64, 48, 40, 64, 1), (250, 199, 2, 0, 0),
                                                          (31, 29, 33, 128, 2)])
def test_queues_equal_wavefront(cuda_device, width, height, spp, threads, ctas, mode):
    base = small_reference_mode(size=24, n=24) if mode == "reference" else small_config_mode(size=24, n=24)
    cfg = base.replace(width=width, height=height)
    vox = volume_for(cfg)
    a = _render(cfg, vox, spp, 0, threads, ctas)
    b = _render(cfg, vox, spp, 1)
    for x, y in zip(a[:3], b[:3]):
        np.testing.assert_array_equal(x, y)
    np.testing.assert_allclose(a[3], b[3], rtol=1e-12, atol=1e-15)   # FP64 atomics in launch order
    assert a[4] == b[4] and a[5] == b[5] == 0


def test_threads_with_different_launch_shapes(cuda_device):
    """Contexts of different launch shapes and majorant grids on one kernel from several threads at once:
    every launch succeeds and gives the single-threaded image."""
    import threading

    cfgs = [small_config_mode(size=24, n=24), small_config_mode(size=24, n=40)]
    jobs = [(cfgs[0], 0), (cfgs[1], 32), (cfgs[0], 96), (cfgs[1], 128)]
    want = [_render(c, volume_for(c), 2, 0, t)[2] for c, t in jobs]
    failed = []

    def work(k):
        try:
            c, t = jobs[k]
            r = Renderer(c.width, c.height)
            setup_scene(r, c, volume=volume_for(c))
            r.set_environment_rgb(constant_environment(c.env_constant if c.env_constant is not None else 0.5))
            r.set_launch_shape(0, t, 0)
            for _ in range(60):
                r.launch_plain(2)
            r.reset_accumulation()
            r.synchronize()
            assert r.device_errors() == 0
            r.close()
        except Exception as e:  # the thread's failure is reported by the test
            failed.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    for (c, t), w in zip(jobs, want):
        np.testing.assert_array_equal(_render(c, volume_for(c), 2, 0, t)[2], w)
