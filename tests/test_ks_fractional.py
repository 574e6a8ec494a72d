"""The KS critical distance for a sample count that is no whole number (an effective
number of dates): the scan takes nslc / 2 as it is, with the library and without it."""

import pytest

from oracle import phase_link as O


@pytest.mark.parametrize("nslc", [0.5, 1.5, 2.9, 10.5, 19.999, 64.25])
@pytest.mark.parametrize("alpha", [0.001, 0.05, 0.5])
def test_fractional_counts(nslc, alpha):
    from dolphin_gb300.shp import ks_critical_distance

    assert ks_critical_distance(nslc, alpha) == O.ks_critical_distance(nslc, alpha)
