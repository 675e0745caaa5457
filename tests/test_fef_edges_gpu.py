"""The ACIS response pass at the edges of its lists and screens: photon counts
around a warp's gathering steps give each photon what a longer list gives it
(everything equal: a photon's result depends on its tag alone), and the error
function is -1 to the last bit wherever the pass takes it to be."""
import numpy as np
import pytest

from test_fef_gpu import case_config, engine, fef_pack  # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu
N = 5000


def _photons(n):
    from marx_gb300 import workloads as W
    from marx_gb300.photons import PhotonList
    full = W.plain_scatter().photons(N, seed=3)
    ph = PhotonList.from_inputs(full.energy[:n].copy(), np.ascontiguousarray(full.p[:, :n]), full.arrival_time[:n].copy())
    ph.tag[:] = np.arange(n, dtype=np.uint32)
    return ph


def _trace(eng, n):
    import torch
    from marx_gb300._native import DevicePhotons
    d = DevicePhotons.from_host(_photons(n))
    eng.trace(d, seed=5)
    torch.cuda.synchronize()
    return d.to_host()


@pytest.mark.parametrize("name", ["fef_acis_i", "qe_acis_i"])
@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, 1023, 1025, 4999])
def test_short_lists_equal_the_long_one(cuda, fef_pack, name, n):  # noqa: F811
    eng = engine(case_config(name), fef_pack)
    a, b = _trace(eng, n), _trace(eng, N)
    for k in ("flags", "ccd_num", "pulse_height", "pi", "y_pixel", "z_pixel"):
        assert np.array_equal(getattr(a, k)[:n], getattr(b, k)[:n]), k
    if n > 1000:
        assert (a.pulse_height > 0).sum() > n // 20


def test_erf_is_minus_one_below_the_screen(cuda):
    """center > 8.5 sigma in float: -center / (sqrt(2) sigma) < -6.01 + 1e-6."""
    import torch
    x = torch.cat([torch.linspace(-6.02, -6.01, 1 << 20, dtype=torch.float64),
                   torch.linspace(-40.0, -6.01, 1 << 20, dtype=torch.float64), torch.tensor([-1e3, -1e30], dtype=torch.float64)])
    assert bool((torch.special.erf(x.cuda()) == -1.0).all())
