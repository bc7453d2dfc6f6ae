"""Replacing a context's volume, on a stand-in for the CUDA runtime (no GPU)."""
import pytest

from . import _fake_cuda, _nvdb

SETTERS = {
    "dense": "lambda r, n: r.set_volume_dense(np.ones((n, n, n), np.float32), 1 / n, [-0.5] * 3)",
    "fbm": "lambda r, n: r.generate_fbm_volume(VolumeSpec(n=n, seed=1, octaves=2), 1 / n, [-0.5] * 3)",
    "union": "lambda r, n: r.generate_fbm_volume(VolumeSpec(n=n, seed=1, octaves=2, union_seed=2), 1 / n, [-0.5] * 3)",
}


@pytest.mark.parametrize("kind", list(SETTERS))
def test_failed_replacement_leaves_the_old_volume_or_none(tmp_path, kind):
    """Memory runs out at any allocation of a replacement: until the old volume's arrays are touched,
    launches go on with it; from then on they are refused until a volume is set, and never see the
    new sizes over the old arrays."""
    out = _fake_cuda.run(f"set_volume = {SETTERS[kind]}\nclouds = {2 if kind == 'union' else 1}\n" + """
for nth in range(1, 12):
    r = Renderer(8, 8)
    r.set_frame(frame_params(C1))
    set_volume(r, 32)
    r.launch_plain(1)
    fake.fake_fail(MALLOC, nth)
    why = failed(lambda: set_volume(r, 80))
    fake.fake_fail(MALLOC, 0)
    launches = fake.fake_calls(LAUNCH)
    refused = failed(lambda: r.launch_plain(1))
    if why is None:  # only the copy for faster lookups is missing
        assert nth > clouds + 4 and refused is None and r.volume_info()["total_leaves"] == 1000
    elif nth <= clouds:
        assert refused is None and r.volume_info()["total_leaves"] == 64, (nth, refused)
    else:
        assert nth <= clouds + 4 and refused and "missing" in refused and fake.fake_calls(LAUNCH) == launches, (nth, refused)
        assert failed(r.volume_info)
    set_volume(r, 80)
    r.launch_plain(1)
    r.close()
print("ok")
""", tmp_path)
    assert out.split() == ["ok"]


@pytest.mark.parametrize("kind", list(SETTERS))
def test_replacement_fits_without_room_for_the_copy(tmp_path, kind):
    """A replacement of the same size needs the volume's arrays and the builder's scratch only: the copy
    of the grid that speeds lookups up gives way to them."""
    out = _fake_cuda.run(f"set_volume = {SETTERS[kind]}\nunion = {kind == 'union'}\n" + """
r = Renderer(8, 8)
empty = fake.fake_bytes()
cells, voxels = 8 ** 3, 4 * 64 ** 3
arrays = voxels + 2 * 4 * cells + 4 * 512          # dense voxels, two tables, one leaf
set_volume(r, 64)
assert fake.fake_bytes() > empty + arrays          # there is a copy
fake.fake_limit(empty + arrays + max(4 * cells, voxels if union else 0))
set_volume(r, 64)
fake.fake_limit(1 << 40)
r.set_frame(frame_params(C1))
r.launch_plain(1)
r.close()
print("ok", fake.fake_bytes())
""", tmp_path)
    assert out.split() == ["ok", "0"]


@pytest.mark.parametrize("kind", list(SETTERS))
def test_replacement_reuses_the_copys_memory(tmp_path, kind):
    """A replacement of like size (a frame of a moving cloud) allocates the volume's own arrays and
    nothing for the copy, reads back the active leaves and the majorant and nothing else; a much smaller
    volume does not keep the large one's copy."""
    out = _fake_cuda.run(f"set_volume = {SETTERS[kind]}\nclouds = {2 if kind == 'union' else 1}\n" + """
r = Renderer(8, 8)
set_volume(r, 64)
held = fake.fake_bytes()
before = [fake.fake_calls(k) for k in (MALLOC, COPY, MEMINFO)]
set_volume(r, 64)
calls = [fake.fake_calls(k) - b for k, b in zip((MALLOC, COPY, MEMINFO), before)]
# voxels of each cloud, active leaves, tables and leaves; copies: the voxels (or a cloud's range), the
# active leaves, the leaf table, the majorant with the copy's size
assert calls == [clouds + 4, clouds + 3, 0], calls
assert fake.fake_bytes() == held
set_volume(r, 16)
small = fake.fake_bytes()
r.close()
r = Renderer(8, 8)
set_volume(r, 16)
assert small == fake.fake_bytes()
print("ok")
""", tmp_path)
    assert out.split() == ["ok"]


def test_cleared_volume_gives_the_copy_back(tmp_path):
    out = _fake_cuda.run("""
r = Renderer(8, 8)
empty = fake.fake_bytes()
r.set_volume_dense(np.ones((64, 64, 64), np.float32), 1 / 64, [-0.5] * 3)
r.clear_volume()
# what stays: dense voxels, two tables, one leaf
assert fake.fake_bytes() - empty == 4 * 64 ** 3 + 2 * 4 * 8 ** 3 + 4 * 512, fake.fake_bytes() - empty
r.set_volume_dense(np.ones((64, 64, 64), np.float32), 1 / 64, [-0.5] * 3)
r.set_frame(frame_params(C1))
r.launch_plain(1)
r.close()
print("ok", fake.fake_bytes())
""", tmp_path)
    assert out.split() == ["ok", "0"]


def test_volume_info_counts_the_copy(tmp_path):
    """The reported bytes are those held for the grid, with the copy and, where there is no room for it,
    without."""
    out = _fake_cuda.run("""
for room in (1 << 40, 0):
    fake.fake_limit(1 << 40)
    r = Renderer(8, 8)
    r.set_volume_dense(np.ones((64, 64, 64), np.float32), 1 / 64, [-0.5] * 3)
    r.clear_volume()
    if not room:
        fake.fake_limit(fake.fake_bytes() + 4 * 8 ** 3)  # the volume's arrays again and the builder's list of cells
    empty = fake.fake_bytes() - (4 * 64 ** 3 + 2 * 4 * 8 ** 3 + 4 * 512)
    r.set_volume_dense(np.ones((64, 64, 64), np.float32), 1 / 64, [-0.5] * 3)
    held = fake.fake_bytes() - empty - 4 * 64 ** 3 - 4 * 512  # without the voxels and the one leaf that no active leaf fills
    assert r.volume_info()["grid_bytes"] == held, (room, r.volume_info(), held)
    assert (held > 2 * 4 * 8 ** 3) == bool(room)
    r.close()
print("ok")
""", tmp_path)
    assert out.split() == ["ok"]


def test_stencil_limit(tmp_path):
    """0 switches the copy off, a limit below its size too, -1 back on; lowering the limit gives a held
    copy back at once; launches go on."""
    out = _fake_cuda.run("""
r = Renderer(8, 8)
r.set_frame(frame_params(C1))
def put(n=64):
    r.set_volume_dense(np.ones((n, n, n), np.float32), 1 / n, [-0.5] * 3)
    r.launch_plain(1)
    return r.volume_info()["grid_bytes"]
plain, copy = 2 * 4 * 8 ** 3, 2 * 4 * 9 ** 3 + 4 * 4096   # tables; the copy's tables and one slot
assert put() == plain + copy
for limit, held in ((0, 0), (copy - 1, 0), (copy, copy), (-1, copy), (1 << 40, copy)):
    r.set_stencil_limit(limit)
    assert put() == plain + held, limit
before = fake.fake_bytes()
r.set_stencil_limit(copy - 1)
assert fake.fake_bytes() == before - copy and r.volume_info()["grid_bytes"] == plain
r.launch_plain(1)
# a copy in a larger one's memory keeps the limit too
r.set_stencil_limit(-1)
put(64)
small = 2 * 4 * 8 ** 3 + 4 * 4096
r.set_stencil_limit(copy)
assert put(56) == 2 * 4 * 7 ** 3 + copy
r.set_stencil_limit(small)
assert put(56) == 2 * 4 * 7 ** 3 + small
assert failed(lambda: r.set_stencil_limit(-2))
r.close()
print("ok", fake.fake_bytes())
""", tmp_path)
    assert out.split() == ["ok", "0"]

def test_failed_copy_is_reported_once(tmp_path):
    out = _fake_cuda.run("""
r = Renderer(8, 8)
r.set_frame(frame_params(C1))
set_volume = lambda: r.set_volume_dense(np.ones((32, 32, 32), np.float32), 1 / 32, [-0.5] * 3)
fake.fake_fail(COPY, 2)
assert failed(set_volume)
fake.fake_fail(COPY, 0)
Renderer(8, 8).close()
set_volume()
r.launch_plain(1)
r.close()
print("ok")
""", tmp_path)
    assert out.split() == ["ok"]


@pytest.mark.parametrize("kind", list(SETTERS) + ["nanovdb"])
def test_failed_calls_leak_nothing(tmp_path, kind):
    """Whichever copy or allocation of a volume's set-up fails, destroying the context gives everything
    back; a query of the free memory that fails costs the stencil copy alone."""
    name = sorted(_nvdb.reference())[0]
    path = _nvdb.fixture_path(name, tmp_path)
    setter = SETTERS.get(kind, f"lambda r, n: r.load_nvdb({str(path)!r})")
    out = _fake_cuda.run(f"set_volume = {setter}\n" + """
for what in (MALLOC, COPY, MEMINFO):
    failures = 0
    for nth in range(1, 16):
        r = Renderer(8, 8)
        r.set_frame(frame_params(C1))
        fake.fake_fail(what, nth)
        why = failed(lambda: set_volume(r, 40))
        fake.fake_fail(what, 0)
        refused = failed(lambda: r.launch_plain(1))
        assert bool(why) == bool(refused), (what, nth, why, refused)
        failures += why is not None
        r.close()
        assert fake.fake_bytes() == 0, (what, nth)
    assert (failures == 0) == (what == MEMINFO)
print("ok")
""", tmp_path)
    assert out.split() == ["ok"]
