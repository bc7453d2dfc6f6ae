"""Host side of the radiance cache on a stand-in for the CUDA runtime (no GPU)."""
import pytest

from . import _fake_cuda


@pytest.mark.parametrize("encoding,records", [(0, 1000), (1, 1000), (2, 100), (2, 1000)])
def test_step_after_a_failed_launch_starts_from_zero(tmp_path, encoding, records):
    """A step whose update is not launched leaves its gradient and loss in the accumulators that the update
    would have cleared; the next step clears them first, and the ones after it have nothing to clear."""
    out = _fake_cuda.run(f"ENC, N = {encoding}, {records}\n" + """
c = nrc.NeuralRadianceCache()
c.initialize(config=nrc.default_config(ENC))
data = np.zeros((N, 14), np.float32)
step = lambda: c.train(0, data.ctypes.data, data.ctypes.data, N)
before = fake.fake_calls(LAUNCH)
step()
launches = fake.fake_calls(LAUNCH) - before
cleared = fake.fake_calls(MEMSET)
step()
assert fake.fake_calls(MEMSET) == cleared
for nth in range(1, launches + 1):
    fake.fake_fail(LAUNCH, nth)
    assert failed(step)
    fake.fake_fail(LAUNCH, 0)
    cleared = fake.fake_calls(MEMSET)
    step()
    after = fake.fake_calls(MEMSET)
    assert after > cleared, nth
    step()
    assert fake.fake_calls(MEMSET) == after
c.finalize()
print("ok", fake.fake_bytes())
""", tmp_path)
    assert out.split() == ["ok", "0"]


@pytest.mark.parametrize("encoding,allocations", [(0, 10), (1, 10), (2, 12)])
def test_creation_allocates_once_for_the_step_accumulators(tmp_path, encoding, allocations):
    """Creating a cache costs an allocation per array (weights, moments, average, accumulators, FP16 images,
    tables, error word) and, with the hash grid, the training features and the workspace."""
    out = _fake_cuda.run(f"ENC = {encoding}\n" + """
before = [fake.fake_calls(k) for k in (MALLOC, MEMSET)]
c = nrc.NeuralRadianceCache()
c.initialize(config=nrc.default_config(ENC))
print(*[fake.fake_calls(k) - b for k, b in zip((MALLOC, MEMSET), before)])
assert np.all(c.gradients() == 0)
c.finalize()
print(fake.fake_bytes())
""", tmp_path)
    assert out.split() == [str(allocations), "5", "0"]
