"""The HRC's double-float forms at their edges, against numpy in double on the
same variates: pulse heights with energies on their branch points and over the
whole range (equal), position blur of each of its three components and of all
(the difference of blurred and unblurred pixels, two single-precision numbers
below 16384 rounded to half an ulp each: 1e-3 pixels), and the exponential of
the Lorentzian's radius.  Fates by the screens of the shield and the Drake flat
are held by the reference's own photons (the HRC fixtures of the parity tests)."""
import ctypes as C

import numpy as np
import pytest

from marx_gb300 import workloads as W
from marx_gb300.photons import PhotonList

pytestmark = pytest.mark.gpu
U_HRC, N_HRC, SEED = 22, 18, 77


def _list(n, seed, arcmin):
    r = np.random.default_rng(seed)
    e = np.exp(r.uniform(np.log(0.06), np.log(10.0), n))
    e[::7], e[1::7], e[2::7], e[3::7] = 0.5, 2.0, np.nextafter(0.5, 1.0), np.nextafter(2.0, 1.0)
    th, ph = np.deg2rad(arcmin / 60.0) * np.sqrt(r.random(n)), r.uniform(0.0, 2 * np.pi, n)
    p = np.stack([-np.cos(th), np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph)])
    q = PhotonList.from_inputs(e, np.ascontiguousarray(p), r.uniform(0.0, 1e4, n))
    q.tag[:] = np.arange(n, dtype=np.uint32)
    return q


@pytest.mark.parametrize("g1,g2,l1", [(1.0, 0.0, 0.0), (0.0, 1.0, 0.0), (0.0, 0.0, 1.0), (1.0, 1.0, 0.2)])
def test_hrc_pulse_heights_and_blur(cuda, g1, g2, l1):
    from marx_gb300._native import Engine
    from oracle.bindings import Oracle
    cfg = W.plain_hrci().cfg
    b = cfg.hrc_i_blur
    b[3], b[7], b[11] = g1, g2, l1
    ph = _list(60_000, 31, 10.0)
    sharp, blurred = ph.copy(), ph.copy()
    cfg.det_ideal = 1
    Engine(cfg).trace_host(sharp, seed=SEED)
    cfg.det_ideal = 0
    Engine(cfg).trace_host(blurred, seed=SEED)
    ok = sharp.good() & blurred.good() & (sharp.y_pixel > 300) & (sharp.z_pixel > 300)
    i = np.flatnonzero(ok)
    assert i.size > 1000
    o = Oracle(W.plain_scatter().cfg)
    u = np.array([[o.philox_uniform(SEED, int(t), U_HRC + k) for k in (2, 3, 4)] for t in ph.tag[i]]).T
    z = np.array([o.philox_normal(SEED, int(t), N_HRC) for t in ph.tag[i]])
    e = ph.energy[i]
    h = np.where(e <= 0.5, 141.582 * np.sqrt(e), np.where(e < 2.0, 107.299 * e ** 0.1, 115.0)) * (1.0 + 0.424661 * z)
    want = np.trunc(np.maximum(h, 0.0)).astype(np.int16)
    assert np.array_equal(blurred.pulse_height[i], want)
    assert np.array_equal(sharp.pulse_height[i], want)
    # the blur in detector pixels (its parameters are quarters of them)
    s1, s2, hw, rmax = 0.42466090014400953 * b[0] / 4, 0.42466090014400953 * b[4] / 4, b[8] / 8, b[12] / 4
    w = np.array([b[3] * 2 * np.pi * s1 ** 2, b[7] * 2 * np.pi * s2 ** 2, b[11] * np.pi * hw ** 2 * np.log1p((rmax / hw) ** 2)])
    w /= w.sum()
    kind = np.where(u[0] < w[0], 0, np.where(u[0] < w[0] + w[1], 1, 2))
    gauss = np.sqrt(-2.0 * np.log(u[1]))
    rad = np.choose(kind, [s1 * gauss, s2 * gauss, hw * np.sqrt(np.expm1(u[1] * np.log1p((rmax / hw) ** 2)))])
    ox = np.array([0.0, (b[5] - b[1]) / 4, (b[9] - b[1]) / 4])[kind]
    oy = np.array([0.0, (b[6] - b[2]) / 4, (b[10] - b[2]) / 4])[kind]
    for col, off in (("y_pixel", ox + rad * np.cos(2 * np.pi * u[2])), ("z_pixel", oy + rad * np.sin(2 * np.pi * u[2]))):
        d = getattr(blurred, col)[i].astype(np.float64) - getattr(sharp, col)[i].astype(np.float64)
        assert np.max(np.abs(d - off)) <= 1.0e-3, col


def test_expm1(cuda):
    """df_expm1 within 2^-42 over the radii's range: seven double-float
    products of 2^-45 each at most, from arguments near 0 to 60."""
    import torch
    from marx_gb300._native import load_library
    L = load_library()
    L.mx_math_check.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_size_t]
    x = np.concatenate([np.geomspace(1e-9, 60.0, 200_000), np.arange(1, 60) * np.log(2.0),
                        np.nextafter(np.arange(1, 60) * np.log(2.0) / 2, 100.0)])
    xd = torch.from_numpy(x).cuda()
    yd = torch.empty_like(xd)
    assert L.mx_math_check(12, xd.data_ptr(), yd.data_ptr(), x.size) == 0
    y = yd.cpu().numpy()
    # the split of x keeps 2^-46 of it: exp(x) - 1 changes by x 2^-46 relative
    assert np.max(np.abs(y / np.expm1(x) - 1.0) / (1.0 + x / 16.0)) <= 2.0 ** -42
