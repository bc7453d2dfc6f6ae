"""The tracker with work queues reading the grid's leaves (no stencil copy: the form a large volume or a
context with a stencil limit of 0 runs) against the same launches through the stencil copy: plain and
logged launches, both majorant modes and stream layouts, meshes in the flat list and through the
BVH, the radiance-cache passes and the frame that combines them.

Both forms draw each path's numbers in the same order and look up the same densities, so volume
scenes are equal to the bit. The mesh kernels' own rounding may differ between two instances of the
kernel, so there the decisions of at least 99.5% of the samples agree (the surface tests' bar), and
the records of those samples to FP32 rounding carried along a path (1e-3)."""
import numpy as np
import pytest

from rtc8_gb300 import nrc
from rtc8_gb300 import surfaces as S
from rtc8_gb300.configs import C_ROOM, C_ROOM_REFERENCE_MODE
from rtc8_gb300.renderer import Renderer, constant_environment, setup_scene

from ._scenes import small_config_mode, small_reference_mode, volume_for

pytestmark = pytest.mark.gpu

SAME = 0.995


def _scene(scene, mode, size):
    if scene == "volume":
        cfg = small_reference_mode(size=size, n=36) if mode == "reference" else small_config_mode(size=size, n=36)
        return cfg, None
    cfg = (C_ROOM_REFERENCE_MODE if mode == "reference" else C_ROOM).replace(width=size, height=size)
    sc = S.room_scene()
    if scene == "spheres":
        sc.add(S.sphere(0.22, 5, 16, 8), S.translation(0.05, 0.05, 0.4))
    return cfg, sc


def _renderer(cfg, surfaces, limit):
    r = Renderer(cfg.width, cfg.height)
    r.set_stencil_limit(limit)
    setup_scene(r, cfg.replace(surfaces=None), volume=volume_for(cfg))
    r.set_environment_rgb(constant_environment(cfg.env_constant))
    if surfaces is not None:
        r.set_surfaces(surfaces)
    return r


def _both(scene, mode, size, work, streams=None):
    cfg, surfaces = _scene(scene, mode, size)
    if streams is not None:
        cfg = cfg.replace(rng_stream_mode=streams)
    out = []
    for limit in (-1, 0):
        r = _renderer(cfg, surfaces, limit)
        info = r.volume_info()
        plain = 4 * 512 * info["active_leaves"] + 8 * info["total_leaves"]
        assert (info["grid_bytes"] > plain) == (limit < 0)  # the two forms are what ran
        out.append(work(r, cfg))
        assert r.device_errors() == 0
        r.close()
    return out


def _agree(same, *pairs):
    """`same`: samples with equal decisions; pairs of per-sample values."""
    assert same.mean() >= SAME, same.mean()
    for a, b in pairs:
        np.testing.assert_allclose(a[same], b[same], rtol=1e-3, atol=1e-6)


@pytest.mark.parametrize("streams", [0, 1])
@pytest.mark.parametrize("mode", ["reference", "config"])
@pytest.mark.parametrize("scene", ["volume", "room", "spheres"])
def test_plain_and_logged_launches(cuda_device, scene, mode, streams):
    import torch

    spp = 3

    def work(r, cfg):
        log = torch.zeros(cfg.width * cfg.height * spp * 4, dtype=torch.int32, device="cuda")
        r.launch_plain_logged(spp, log.data_ptr())
        r.synchronize()
        logged = r.download_sum()[0]
        r.reset_accumulation()
        r.launch_plain(spp)
        r.synchronize()
        return log.cpu().numpy().reshape(-1, 4 * spp), logged, r.download_sum()[0], r.rng_states()

    a, b = _both(scene, mode, 48, work, streams)
    if scene == "volume":
        for x, y in zip((a[0], a[3]), (b[0], b[3])):
            np.testing.assert_array_equal(x, y)
        for k in (1, 2):  # FP64 atomics in launch order
            np.testing.assert_allclose(a[k], b[k], rtol=1e-12, atol=1e-15)
    else:
        same = (a[0] == b[0]).all(axis=1)
        _agree(same, (a[1].reshape(-1, 3), b[1].reshape(-1, 3)))
        np.testing.assert_allclose(a[2].sum(), b[2].sum(), rtol=2e-2)


@pytest.mark.parametrize("mode", ["reference", "config"])
@pytest.mark.parametrize("scene", ["volume", "room", "spheres"])
def test_radiance_cache_render_pass(cuda_device, scene, mode):
    import torch

    def work(r, cfg):
        r.nrc_set_query_density(True)
        r.nrc_set_termination_factor(0.02)
        r.launch_render_nrc()
        torch.cuda.synchronize()
        v = {k: t.cpu().numpy() for k, t in r.nrc_views().items()}
        bits = v["infer_terminal"][:, 3].copy().view(np.uint32)
        n = cfg.width * cfg.height
        return bits, v["infer_terminal"][:, :3], v["infer_query"][:n], v["frame_contribution"], r.rng_states()

    a, b = _both(scene, mode, 48, work)
    has = (a[0] & 1) == 1
    assert has.any()
    if scene == "volume":
        for k in (0, 4):
            np.testing.assert_array_equal(a[k], b[k])
        for x, y in ((a[1], b[1]), (a[2][has], b[2][has]), (a[3], b[3])):
            np.testing.assert_array_equal(x.view(np.uint32), y.view(np.uint32))
    else:
        _agree((a[0] == b[0]) & (a[4] == b[4]), (a[1], b[1]), (a[3], b[3]))


@pytest.mark.parametrize("scene", ["volume", "room", "spheres"])
def test_radiance_cache_training_pass(cuda_device, scene):
    """Training vertices lie in the order their paths reached them: the records are compared sorted."""
    import torch

    def work(r, cfg):
        r.nrc_set_query_density(True)
        r.nrc_set_termination_factor(0.02)
        r.prepare_nrc(0, 2654435761, True)
        r.launch_generate_training(0)
        torch.cuda.synchronize()
        v = {k: t.cpu().numpy() for k, t in r.nrc_views().items()}
        count = int(v["counters"][0])
        rec = np.concatenate([v["train_query0"][:count], v["train_target0"][:count], v["train_vertex"][:count, :3]], axis=1)
        return count, rec, v["train_rng"]

    a, b = _both(scene, "reference", 64, work)
    assert a[0] > 0
    if scene == "volume":
        assert a[0] == b[0]
        ra, rb = (x.view(np.uint32) for x in (a[1], b[1]))
        np.testing.assert_array_equal(ra[np.lexsort(ra.T)], rb[np.lexsort(rb.T)])
        np.testing.assert_array_equal(a[2], b[2])
    else:
        assert (a[2] == b[2]).mean() >= SAME
        assert abs(a[0] - b[0]) <= 0.02 * a[0]


@pytest.mark.parametrize("scene", ["volume", "room", "spheres"])
def test_combined_frame(cuda_device, scene):
    """A frame whose training and render paths share one launch; the render records do not depend on
    the network."""
    import torch

    def work(r, cfg):
        r.nrc_set_query_density(True)
        r.nrc_set_termination_factor(0.02)
        cache = nrc.NeuralRadianceCache()
        cache.initialize(config=nrc.default_config(nrc.NRC_ENCODING_VOLUME))
        r.nrc_frame(cache, 2, 3, True)
        torch.cuda.synchronize()
        v = {k: t.cpu().numpy() for k, t in r.nrc_views().items()}
        assert cache.device_errors() == 0
        cache.finalize()
        bits = v["infer_terminal"][:, 3].copy().view(np.uint32)
        n = 3 * cfg.width * cfg.height
        return bits, v["infer_terminal"][:, :3], v["infer_query"][:n], v["frame_contribution"]

    a, b = _both(scene, "config", 48, work)
    has = (a[0] & 1) == 1
    assert has.any()
    if scene == "volume":
        np.testing.assert_array_equal(a[0], b[0])
        for x, y in ((a[1], b[1]), (a[2][has], b[2][has]), (a[3], b[3])):
            np.testing.assert_array_equal(x.view(np.uint32), y.view(np.uint32))
    else:
        _agree(a[0] == b[0], (a[1], b[1]), (a[3], b[3]))
