"""Extended sources given a direction that is not of unit length (one widened
from single precision is off by some 1e-8): the photons' directions are unit
vectors all the same, on both sides of the size up to which a source takes
the small-angle form, and those of the unit vector along it."""
import numpy as np
import pytest

from marx_gb300 import batched as B

from test_sources_gpu import generate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,param", [("GAUSS", (2.0,)), ("GAUSS", (900.0,)), ("DISK", (0.0, 5.0)),
                                        ("DISK", (0.0, 2000.0)), ("BETA", (3.0, 0.7)), ("BETA", (300.0, 0.7))])
def test_directions_are_unit_vectors(cuda, kind, param):
    from marx_gb300._native import Engine
    n, seed, th, ph = 20_000, 77, 0.004, 0.7
    unit = np.array([-np.cos(th), np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph)])
    eng = Engine(B.batched_config())
    want = generate(eng, B.make_source(unit, kind, param, energy=(0.5, 7.0), num_photons=n), n, seed).p
    for p in (unit * (1 + 3e-8), unit * (1 - 3e-8), unit * 1.25):
        q = generate(eng, B.make_source(p, kind, param, energy=(0.5, 7.0), num_photons=n), n, seed).p
        # a handful of ulps of 1, as for a direction of unit length
        assert np.max(np.abs(np.sqrt((q.astype(np.longdouble) ** 2).sum(0)) - 1)) < 1e-15
        assert np.max(np.abs(q - want)) < 1e-15
