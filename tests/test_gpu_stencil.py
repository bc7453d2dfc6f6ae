"""The tracker's lookups through the stencil copy of the grid against lookups through its leaves.

The wavefront tracker reads the 8^3 leaves; the persistent tracker reads the stencil copy. Both
draw each path's random numbers in the same order, so their decision logs, RNG states and sums are
equal to the bit wherever the two layouts give the same densities: grids smaller than a leaf, one
voxel past a leaf, partial leaves on each axis, empty leaves next to full ones (stencils that
straddle them), a single voxel at a corner, an empty grid."""
import numpy as np
import pytest

from rtc8_gb300.configs import VolumeSpec
from rtc8_gb300.renderer import constant_environment

from ._scenes import small_config_mode, small_reference_mode
from .test_gpu_plain import _gpu_logged

pytestmark = pytest.mark.gpu


def _voxels(dims, fill):
    rng = np.random.default_rng(sum(dims))
    v = rng.random(dims).astype(np.float32)
    if fill == "blocks":  # whole leaves and single voxel planes set to zero
        keep = rng.random(tuple((d + 7) // 8 for d in dims)) < 0.5
        v *= np.kron(keep, np.ones((8, 8, 8)))[: dims[0], : dims[1], : dims[2]].astype(np.float32)
        v[dims[0] // 2] = 0.0
    elif fill == "corner":
        v[:] = 0.0
        v[-1, -1, -1] = 1.0
        v[0, 0, 0] = 0.5
    elif fill == "empty":
        v[:] = 0.0
    return v


@pytest.mark.parametrize("mode", ["reference", "config"])
@pytest.mark.parametrize("dims,fill", [((2, 2, 2), "full"), ((8, 8, 8), "full"), ((9, 17, 16), "full"),
                                       ((33, 7, 25), "blocks"), ((48, 40, 56), "blocks"), ((16, 24, 9), "corner"),
                                       ((12, 12, 12), "empty")])
def test_stencil_lookups_equal_leaf_lookups(cuda_device, dims, fill, mode):
    vox = _voxels(dims, fill)
    base = small_reference_mode(size=24) if mode == "reference" else small_config_mode(size=24)
    cfg = base.replace(volume=VolumeSpec(n=max(dims), seed=1, octaves=1, sigma_t_max=20.0))
    env = constant_environment(cfg.env_constant if cfg.env_constant is not None else 0.5)
    a = _gpu_logged(cfg, vox, env, 4, tracker=0)
    b = _gpu_logged(cfg, vox, env, 4, tracker=1)
    np.testing.assert_array_equal(a["log"], b["log"])
    np.testing.assert_array_equal(a["rng"], b["rng"])
    np.testing.assert_array_equal(a["mean"], b["mean"])
    np.testing.assert_allclose(a["sum"], b["sum"], rtol=1e-12, atol=1e-15)   # FP64 atomics in launch order
    assert a["counters"] == b["counters"] and a["errors"] == b["errors"] == 0
