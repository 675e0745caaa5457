"""ACIS response tables with values at the edges of what a file may hold: a
gaussian of NaN width is left out, as one of zero width is, and amplitudes so
small that the areas leave the range of normal floats give what amplitudes of
one give (only their ratios count).  Both compared draw for draw."""
import numpy as np
import pytest

from marx_gb300.caldb.pack import DEFAULT_PACK, pack_with_fef, read_pack, write_pack

from test_fef_edges_gpu import N, _trace
from test_fef_gpu import CONTAM_FILE, FEF_FILE, case_config, engine

pytestmark = pytest.mark.gpu
FWHM, POS, AMP = range(3)


@pytest.fixture(scope="module")
def sections(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("fef") / "fef.mxpack")
    pack_with_fef(DEFAULT_PACK, FEF_FILE, out, contam_path=CONTAM_FILE)
    return read_pack(out)


def _pulse_heights(sections, path, change):
    S = dict(sections)
    v = S["acis/fef/vals"].copy()
    change(v[:, 2:].reshape(v.shape[0], -1, 3))       # [row][gaussian][FWHM, POS, AMP]
    S["acis/fef/vals"] = v
    write_pack(str(path), S)
    eng = engine(case_config("fef_acis_i"), str(path))
    q = _trace(eng, N)
    assert eng.overrun_count() == 0
    return q


@pytest.mark.parametrize("g", [0, 1, 2])
def test_nan_width_leaves_the_gaussian_out(cuda, sections, tmp_path, g):
    def width(value):
        def change(t):
            t[:, g, FWHM] = value
        return change
    a = _pulse_heights(sections, tmp_path / "zero.mxpack", width(0.0))
    b = _pulse_heights(sections, tmp_path / "nan.mxpack", width(np.nan))
    for k in ("flags", "pulse_height", "pi"):
        assert np.array_equal(getattr(a, k), getattr(b, k)), k
    assert (a.pulse_height > 0).sum() > 100


def test_areas_below_a_normal_float(cuda, sections, tmp_path):
    """One gaussian of sigma 100 centred half a sigma below zero: 31 % of its
    area above zero, 2^-126.7 for an amplitude of 2^-133, 69 % below, 2^-125.5."""
    def amplitude(value):
        def change(t):
            t[:] = 0.0
            t[:, 0] = [100.0 * np.sqrt(8 * np.log(2.0)), -50.0, value]
        return change
    a = _pulse_heights(sections, tmp_path / "one.mxpack", amplitude(1.0))
    b = _pulse_heights(sections, tmp_path / "small.mxpack", amplitude(2.0 ** -133))
    for k in ("flags", "pulse_height", "pi"):
        assert np.array_equal(getattr(a, k), getattr(b, k)), k
    assert (a.pulse_height > 0).sum() > 100
