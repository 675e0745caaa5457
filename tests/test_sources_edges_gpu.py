"""GAUSS and DISK source photons on both sides of the size that the
double-float form takes (2^-10 rad; GAUSS sigma of 0.4 of it), against the
models' formulas in long double on the same draws."""
import numpy as np
import pytest

from marx_gb300 import batched as B

from test_sources_gpu import generate

pytestmark = pytest.mark.gpu
ARCSEC = np.pi / 648000.0


def draws(seed, n, slot):
    """Uniform draw `slot` of photons 0..n-1 (Philox4x32-10)."""
    m = np.uint64(0xFFFFFFFF)
    c = [np.arange(n, dtype=np.uint64), np.full(n, slot, np.uint64), np.full(n, 0x5A5A0003, np.uint64), np.zeros(n, np.uint64)]
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        a, b = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(b >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), b & m, (a >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), a & m]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return ((c[0] << np.uint64(21)) | (c[1] >> np.uint64(11))).astype(np.longdouble) * np.longdouble(2) ** -53


@pytest.mark.parametrize("kind,param", [("GAUSS", (1e-3,)), ("GAUSS", (2.0,)), ("GAUSS", (80.0,)), ("GAUSS", (81.0,)),
                                        ("GAUSS", (900.0,)), ("DISK", (0.0, 5.0)), ("DISK", (150.0, 201.0)),
                                        ("DISK", (10.0, 202.0)), ("DISK", (0.0, 2000.0))])
def test_directions_either_side_of_the_small_angle_form(cuda, kind, param):
    from marx_gb300._native import Engine
    n, seed = 20_000, 0x123456789
    th, ph = 0.004, 0.7
    p = np.array([-np.cos(th), np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph)])
    q = generate(Engine(B.batched_config()), B.make_source(p, kind, param, energy=(0.5, 7.0), num_photons=n), n, seed)
    f = np.longdouble
    pl = p.astype(f)
    pn = np.array([-pl[1] / pl[0], f(1), f(0)])
    pn = pn / np.sqrt((pn * pn).sum())
    phi, u = 2 * f("3.14159265358979323846264338327950288") * draws(seed, n, 1), draws(seed, n, 2)
    if kind == "GAUSS":
        ang = f(param[0] * ARCSEC) * np.sqrt(-np.log(u))
    else:
        t1, r = f(param[1] * ARCSEC), (f(param[0]) / f(param[1])) ** 2
        ang = t1 * np.sqrt(r + (1 - r) * u)
    w = np.cross(pn, pl)
    ref = np.cos(ang) * pl[:, None] + np.sin(ang) * (np.cos(phi) * w[:, None] + np.sin(phi) * pn[:, None])
    # unit vectors formed by a few roundings: a handful of ulps of 1
    assert np.max(np.abs(q.p - ref)) < 1e-15
