"""Observed traces with an infinite sample: the gather's scales become infinite,
and every kind gives a value where the oracle has one, and none where it has none."""
import numpy as np
import pytest

from oracle import pyoracle as po
from tests.test_ot import TOL, _gather
from tests.test_ot_formats import _fn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [1, 2, 3])
@pytest.mark.parametrize("value", [np.inf, -np.inf])
@pytest.mark.parametrize("nt", [500, 7300])
def test_infinite_scale_of_a_gather(kind, value, nt):
    obs_x, obs_z, cal_x, cal_z = _gather(5, 4, nt)
    obs_z[2, 77] = value
    m_ref, rx_ref, rz_ref = po.ot_gather(kind, 1e-3, obs_x, obs_z, cal_x, cal_z)
    rx, rz, m = _fn(kind)(obs_x, obs_z, cal_x, cal_z, 1e-3)
    assert np.isnan(m) and np.isnan(m_ref)
    assert np.array_equal(np.isnan(rz), np.isnan(rz_ref)) and not np.isnan(rx).any()
    ok = ~np.isnan(rz_ref)
    assert np.linalg.norm(rz[ok] - rz_ref[ok]) <= TOL * np.linalg.norm(rz_ref[ok])
    assert np.linalg.norm(rx - rx_ref) <= TOL * np.linalg.norm(rx_ref)
