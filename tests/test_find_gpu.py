"""The index tables of the interpolation abscissae against the bisection they
stand for: the same index for every abscissa, the floats next to it, points
between, and values outside, on the calibration's own tables and on shapes
that a table may have (uniform, logarithmic, repeated values, clusters, too
short, unordered).  No tolerance: the indices are equal."""
import ctypes as C
import struct

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tables():
    from marx_gb300.caldb.pack import DEFAULT_PACK
    b = open(DEFAULT_PACK, "rb").read()
    out = {}
    for i in range(struct.unpack_from("<I", b, 8)[0]):
        name, dt, nd, *rest = struct.unpack_from("<48sII4QQQ", b, 16 + 104 * i)
        name = name.rstrip(b"\0").decode()
        if dt == 0 and name.split("/")[0] in ("hrma", "hetg", "letg", "grating", "hrc", "acis") and "subpix" not in name:
            a = np.frombuffer(b, "<f4", rest[5] // 4, rest[4]).reshape(rest[:nd])
            if a.ndim == 1 or "eff" not in name:
                out[name] = np.array(a if a.ndim == 1 else a[0])
    rng = np.random.default_rng(3)
    out["uniform"] = np.linspace(0.05, 10.0, 5000, dtype=np.float32)
    out["log"] = np.geomspace(1e-20, 1e20, 777).astype(np.float32)
    out["repeats"] = np.repeat(np.linspace(0.1, 1.0, 100, dtype=np.float32), rng.integers(1, 5, 100))
    out["cluster"] = np.sort(np.concatenate([1.0 + 1e-7 * np.arange(40), np.linspace(0.1, 9, 60)])).astype(np.float32)
    out["short"] = np.array([0.5, 1.0, 2.0], dtype=np.float32)
    out["eight"] = np.arange(1, 9).astype(np.float32)
    out["from zero"] = np.linspace(0.0, 1.0, 50, dtype=np.float32)
    out["one value"] = np.full(20, 2.0, dtype=np.float32)
    out["unordered"] = rng.random(300).astype(np.float32) + 0.1
    out["65535"] = np.linspace(1.0, 2.0, 65535, dtype=np.float32)
    out["too many"] = np.linspace(1.0, 3.0, 65536, dtype=np.float32)
    return out


@pytest.mark.parametrize("name", sorted(_tables()))
def test_index_table_equals_bisection(cuda, name):
    import torch
    from marx_gb300._native import load_library
    L = load_library()
    L.mx_math_check.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_size_t]
    x = _tables()[name].astype(np.float64)
    xd = torch.from_numpy(x).cuda()
    yd = torch.full((x.size,), -1.0, dtype=torch.float64, device="cuda")
    assert L.mx_math_check(11, xd.data_ptr(), yd.data_ptr(), x.size) == 0
    assert (yd.cpu().numpy() == 0.0).all()
