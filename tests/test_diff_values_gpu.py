"""Weighted rays through a mirror whose optical constants are NaN at the ray
energy: a weight that is not a number adds nothing to the image."""
import numpy as np
import pytest

from marx_gb300.caldb.pack import DEFAULT_PACK, read_pack, write_pack
from marx_gb300.diff import FRESH, NPARAM, DiffImage, diff_mirror_config, diff_workload

pytestmark = pytest.mark.gpu


def test_nan_weights_leave_the_image_empty(cuda, tmp_path):
    from marx_gb300._native import Engine
    S = read_pack(DEFAULT_PACK)
    S["hrma/optconst"] = S["hrma/optconst"].copy()
    S["hrma/optconst"][1] = np.nan
    pack = str(tmp_path / "nan.mxpack")
    write_pack(pack, S)
    eng = Engine(diff_mirror_config(ideal=False), pack=pack)
    d = DiffImage(eng, diff_workload(n_rays=5000).cfg)
    theta = np.zeros(NPARAM)
    w = d.rays(theta, FRESH)[2]
    assert bool(w.isnan().any()) and not bool((w > 0).any())
    assert float(d.forward(theta, FRESH).abs().max()) == 0.0
    d.close()
