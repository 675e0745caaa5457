"""Index tables of abscissae that crowd together: thousands of values in what
would be one cell, a lone small value ahead of a dense table, the calibration's
own tables of the LETG and the ACIS.  Every lookup finds the bisection's index
with no more loads than it takes (the check counts both)."""
import ctypes as C

import numpy as np
import pytest

from test_find_gpu import _tables

pytestmark = pytest.mark.gpu


def _crowded():
    r = np.random.default_rng(8)
    out = {k: v for k, v in _tables().items() if k in ("letg/geff0/energy", "acis/qe0", "acis/qe5", "hrma/optconst", "eight")}
    out["one cell"] = np.sort(np.concatenate([1.0 + 2.4e-7 * np.arange(4000), np.geomspace(1e-6, 1e6, 50)])).astype(np.float32)
    out["lone value ahead"] = np.concatenate([[1e-30], np.linspace(1.0, 1.5, 3000)]).astype(np.float32)
    out["two crowds"] = np.sort(np.concatenate([r.normal(0.3, 1e-4, 500), r.normal(7.0, 1e-3, 500)])).astype(np.float32)
    out["long run of equal values"] = np.sort(np.concatenate([np.full(300, 2.0), np.linspace(1, 3, 300)])).astype(np.float32)
    for n in (8, 9, 16, 17, 64, 65):
        out[f"{n} values"] = np.linspace(0.5, 4.0, n, dtype=np.float32)
    return out


@pytest.mark.parametrize("name", sorted(_crowded()))
def test_lookups_cost_no_more_than_a_bisection(cuda, name):
    import torch
    from marx_gb300._native import load_library
    L = load_library()
    L.mx_math_check.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_size_t]
    x = _crowded()[name].astype(np.float64)
    xd = torch.from_numpy(x).cuda()
    yd = torch.full((x.size,), -1.0, dtype=torch.float64, device="cuda")
    assert L.mx_math_check(11, xd.data_ptr(), yd.data_ptr(), x.size) == 0
    assert (yd.cpu().numpy() == 0.0).all()
