"""Launch shapes the batch's autotuner tries by default (no GPU)."""
from rtc8_gb300.batch import LAUNCH_CANDIDATES


def test_default_candidates_are_different_launches():
    """The tracker with work queues takes its CTAs per SM from a candidate and ignores the park threshold,
    which leaf staging alone reads: no two candidates may be the same launch."""
    assert len({ctas for ctas, _ in LAUNCH_CANDIDATES}) == len(LAUNCH_CANDIDATES) > 1
    assert (0, 0) in LAUNCH_CANDIDATES and all(park == 0 for _, park in LAUNCH_CANDIDATES)
    # The default (0) is as many CTAs of 128 threads as fit, 6 of the volume kernels.
    assert all(ctas < 6 for ctas, _ in LAUNCH_CANDIDATES)
