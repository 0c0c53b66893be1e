"""The number formats of the OT kernel (csrc/sfwi_ot.cu): integer CDFs and float
pairs, with FP64 at scales that floats do not cover.  The oracle works in FP64;
the weights are FP32 exponentials, hence the tolerance of the other OT tests."""
import numpy as np
import pytest

from oracle import pyoracle as po
from tests.test_ot import TOL, _gather

pytestmark = pytest.mark.gpu


def _fn(kind):
    import sfwi_gb300 as sg
    return {1: sg.OT, 2: sg.OT_power, 3: sg.OT_alltrace}[kind]


@pytest.mark.parametrize("kind", [1, 2, 3])
@pytest.mark.parametrize("ntr,nt,scale,ratio", [
    (2, 1, 1.0, 1.0), (2, 2, 1.0, 1.0), (3, 33, 1.0, 1.0), (300, 9, 1.0, 1.0), (257, 290, 1.0, 1.0),
    (3, 400, 1e-22, 1.0), (3, 400, 1e-16, 1.0), (3, 400, 1e-14, 1.0), (3, 400, 1e14, 1.0), (3, 400, 1e16, 1.0),
    (2, 4096, 1.0, 30.0), (2, 4097, 1.0, 1e-4), (2, 8001, 1e-16, 1.0), (3, 700, 1.0, 1e8),
])
def test_ot_at_edges_of_its_formats(kind, ntr, nt, scale, ratio):
    """lengths at the edges of a run, a power of two and the scratch form;
    amplitudes on both sides of the line to FP64; predictions far larger or
    smaller than the data"""
    obs_x, obs_z, cal_x, cal_z = (np.float32(scale) * a for a in _gather(nt, ntr, nt, shift=min(6, nt // 2)))
    cal_x, cal_z = np.float32(ratio) * cal_x, np.float32(ratio) * cal_z
    m_ref, rx_ref, rz_ref = po.ot_gather(kind, 1e-3, obs_x, obs_z, cal_x, cal_z)
    rx, rz, m = _fn(kind)(obs_x, obs_z, cal_x, cal_z, 1e-3)
    for a, b in ((rx, rx_ref), (rz, rz_ref)):
        assert np.linalg.norm(a.astype(np.float64) - b) <= TOL * np.linalg.norm(b.astype(np.float64))
    assert abs(m - m_ref) <= TOL * abs(m_ref)


@pytest.mark.parametrize("kind", [1, 2, 3])
def test_ot_vanishes_on_equal_traces(kind):
    obs_x, obs_z, _, _ = _gather(3, 4, 3000)
    rx, rz, m = _fn(kind)(obs_x, obs_z, obs_x, obs_z, 1e-3)
    assert m == 0 and not rx.any() and not rz.any()


@pytest.mark.parametrize("kind", [1, 2])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_ot_keeps_a_bad_trace_to_itself(kind, value):
    obs_x, obs_z, cal_x, cal_z = _gather(5, 4, 500)
    rx0, rz0, _ = _fn(kind)(obs_x, obs_z, cal_x, cal_z, 1e-3)
    cal_z[2, 77] = value
    rx, rz, m = _fn(kind)(obs_x, obs_z, cal_x, cal_z, 1e-3)
    assert np.isnan(m) and np.isnan(rz[2]).all()
    keep = [0, 1, 3]
    assert np.array_equal(rz[keep], rz0[keep]) and np.array_equal(rx, rx0)
