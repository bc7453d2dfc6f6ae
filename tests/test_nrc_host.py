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
    assert after - cleared == 2, (nth, after - cleared)
    step()
    assert fake.fake_calls(MEMSET) == after
c.finalize()
print("ok", fake.fake_bytes())
""", tmp_path)
    assert out.split() == ["ok", "0"]
