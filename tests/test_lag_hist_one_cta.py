"""The shape with one CTA per SM pays for many taus only: fewer stay on the ring kernel (launches of one batch) or
on launches of one batch (launches of two). CPU, through tests/hist_shape_probe.cu."""
import pytest

from cuda_multiddm_b200.media import log_taus
from test_lag_hist_shape import probe, run  # noqa: F401


@pytest.mark.parametrize("last,count,single,pair", [
    (1000, 48, True, True),    # two and three CTAs per SM
    (1300, 48, True, False),   # one CTA per SM for two batches
    (1000, 64, True, False), (1500, 64, True, False), (1000, 80, True, False),
    (1000, 100, True, True),
    (1300, 100, False, None), (1650, 80, False, None),  # and for one
    (1000, 128, True, True), (1650, 200, True, True),
])
def test_lists_on_one_cta_per_sm(probe, last, count, single, pair):  # noqa: F811
    taus = log_taus(1, last, count)
    shapes = run(probe, [(False, 32, last + 64, 10 ** 6, 32, taus)])[0]
    assert (shapes[0][0] > 0) == single
    if pair is not None:
        assert (shapes[1][0] > 0) == pair
