"""The front half of the trace where its single-precision and fixed-point
steps meet the double-precision ones: conversions and azimuths against
their bounds, the dither's sines at the edges of their range, and photons
far off axis and through turned paraboloids against the CPU oracle."""
import ctypes as C
import os

import numpy as np
import pytest

from marx_gb300 import workloads as W
from marx_gb300.caldb.pack import DEFAULT_PACK, read_pack, write_pack
from marx_gb300.photons import PhotonList

pytestmark = pytest.mark.gpu


def _check(fn, x, width=1):
    import torch
    from marx_gb300._native import load_library
    L = load_library()
    L.mx_math_check.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_size_t]
    xd = torch.from_numpy(np.ascontiguousarray(x, dtype=np.float64)).cuda()
    yd = torch.empty(x.size * width, dtype=torch.float64, device="cuda")
    assert L.mx_math_check(fn, xd.data_ptr(), yd.data_ptr(), x.size) == 0
    return yd.cpu().numpy()


def test_split_and_join(cuda):
    """hi + lo holds 47 bits of a double (truncated high part, rounded low
    part), and a float comes back as it went in."""
    r = np.random.default_rng(3)
    x = r.uniform(-1, 1, 20000) * np.exp2(r.integers(-40, 20, 20000).astype(float))
    p = np.exp2(np.arange(-50, 40).astype(float))
    x = np.concatenate([x, p, -p, np.nextafter(p, 0), np.nextafter(p, np.inf), [0.0, 1 - 2.0 ** -53, 2.0 ** -70, -1e30]])
    y = _check(9, x)
    near = np.abs(x) < 2.0 ** 59
    assert np.all(np.abs(y - x)[near] <= 2.0 ** -46 * np.abs(x)[near])
    assert np.all(np.abs(y - x)[~near] <= 2.0 ** -23 * np.abs(x)[~near])
    f = x.astype(np.float32).astype(np.float64)
    assert np.array_equal(_check(9, f), f)


def test_azimuth_within_two_to_minus_45(cuda):
    r = np.random.default_rng(4)
    x = np.concatenate([r.random(20000), np.arange(64) / 64.0, np.nextafter(np.arange(1, 64) / 64.0, 0),
                        [0.0, 2.0 ** -53, 1 - 2.0 ** -53, 2.0 ** -70, 5e-324, 0.125 + 2.0 ** -40]])
    y = _check(10, x, 2).reshape(-1, 2)
    a = 2 * np.longdouble("3.14159265358979323846264338327950288") * (x.astype(np.longdouble) - np.longdouble(0.125))
    assert np.max(np.abs(y[:, 0] - np.sin(a))) < 2.0 ** -45
    assert np.max(np.abs(y[:, 1] - np.cos(a))) < 2.0 ** -45


@pytest.mark.parametrize("period", [1000.0, 4.0, 0.5, 3.7e7])
def test_dither_offsets_round_like_the_double_expression(cuda, period):
    """Times of no, a tiny, many and too many quarter turns (2^12 is the
    fixed-point form's limit), and before zero."""
    from marx_gb300._native import Engine
    cfg = W.plain_scatter().cfg
    cfg.dither_period[:] = [period, period * 0.707, 1e5]
    r = np.random.default_rng(5)
    q = period / 4
    t = np.concatenate([[0.0, -0.0, 5e-324, 1e-300, 1e-12, -1e-12], q * np.arange(1, 60), q * (2.0 ** 12 + np.arange(-3, 4)),
                        q * np.exp(r.uniform(-30, np.log(3e5), 4000)), -q * r.uniform(0, 500, 500)])
    p = np.zeros((3, t.size)); p[0] = -1.0
    ph = PhotonList.from_inputs(np.ones(t.size), p, t)
    Engine(cfg).trace_host(ph, stages=1, seed=1)
    for k in range(2):
        amp = cfg.dither_amp[k] * (np.pi / (180.0 * 3600))
        v = amp * np.sin((2.0 * np.pi) * t / cfg.dither_period[k])
        f = v.astype(np.float32)
        # a float away only where the double lies within two of its ulps (two
        # libraries' sines) of the boundary between the two floats
        other = ph.dither_state[k].astype(np.float64)
        mid = 0.5 * (other + f.astype(np.float64))
        assert np.all((ph.dither_state[k] == f) | (np.abs(v - mid) <= 2 * np.spacing(np.abs(v)))), period


def _against_oracle(cfg, ph, pack=None, seed=9, positions=True):
    from marx_gb300._native import Engine
    from oracle.bindings import Oracle
    q, o = ph.copy(), ph.copy()
    Engine(cfg, pack=pack).trace_host(q, seed=seed)
    Oracle(cfg, pack).trace(o, seed=seed, threads=os.cpu_count() or 1)
    for c in ("flags", "mirror_shell", "ccd_num"):
        np.testing.assert_array_equal(getattr(q, c), getattr(o, c), err_msg=c)
    if not positions:
        return
    assert np.max(np.abs(q.x - o.x)) < 1e-9
    assert np.max(np.abs(q.p - o.p)) < 1e-12


@pytest.mark.parametrize("n", [50_000, 100_001])
def test_far_off_axis_photons(cuda, n):
    """Rays up to 45 arcmin off axis, where the ray meets the paraboloid
    almost along its surface: the miss screen changes no photon's fate.
    (Positions there depend on the order of roundings: an intersection of a
    ray at a hundredth of a degree to the surface turns the last bit of the
    squared radius, 6e-11 mm^2, into more than 1e-9 mm along it.)"""
    w = W.plain_scatter()
    r = np.random.default_rng(6)
    ph = PhotonList.from_inputs(r.uniform(0.3, 8, n), W.offaxis_directions(r.uniform(0, 45, n) * W.ARCMIN,
                                                                         r.uniform(0, 2 * np.pi, n)), r.uniform(0, 1e4, n))
    _against_oracle(w.cfg, ph, positions=False)


def test_turned_paraboloids(cuda, tmp_path):
    """A calibration whose paraboloids are turned, unlike the stock one."""
    S = read_pack(DEFAULT_PACK)
    rdb = S["hrma/rdb"].reshape(2, 4, 9)
    rdb[0, :, 6] = [0.001, -0.002, 0.0015, 0.0005]
    rdb[0, :, 7] = [-0.0008, 0.001, 0.0, 0.002]
    S["hrma/rdb"] = rdb.reshape(S["hrma/rdb"].shape)
    pack = str(tmp_path / "turned.mxpack")
    write_pack(pack, S)
    w = W.plain_scatter()
    _against_oracle(w.cfg, w.photons(70_000, seed=8), pack=pack)


@pytest.mark.parametrize("blur,scat,emin,emax", [(30.0, 1.0, 0.3, 8.0),      # blur angles past the series' 2e-5 rad
                                                 (0.3, 40.0, 0.3, 8.0),      # scattering past its 2^-10 rad
                                                 (0.0, 1.0, 0.02, 12.0),     # energies outside the tables' rows
                                                 (0.3, 0.0, 0.3, 8.0)])      # no scattering angle at all
def test_reflections_at_the_edges_of_their_series(cuda, blur, scat, emin, emax):
    """Blur and scattering on both sides of the angles their double-float
    forms take: every photon's fate, and where the survivors arrive."""
    from marx_gb300._native import Engine
    from oracle.bindings import Oracle
    w = W.plain_scatter()
    for k in range(4):
        w.cfg.blur_p[k] = w.cfg.blur_h[k] = blur
        w.cfg.scat_p[k] *= scat
        w.cfg.scat_h[k] *= scat
    n, r = 70_000, np.random.default_rng(10)
    ph = w.photons(n, seed=10)
    ph.energy[:] = np.exp(r.uniform(np.log(emin), np.log(emax), n))
    q, o = ph.copy(), ph.copy()
    Engine(w.cfg).trace_host(q, seed=11)
    Oracle(w.cfg).trace(o, seed=11, threads=os.cpu_count() or 1)
    for c in ("flags", "mirror_shell", "ccd_num"):
        np.testing.assert_array_equal(getattr(q, c), getattr(o, c), err_msg=c)
    good = q.good()
    assert good.sum() > 1000
    assert np.max(np.abs(q.x - o.x)[:, good]) < 1e-9
    assert np.max(np.abs(q.p - o.p)[:, good]) < 1e-12


@pytest.mark.parametrize("scat", [1.0, 30.0])
def test_photons_left_for_later_equal_the_fused_trace(cuda, scat):
    """A list long enough for phases B and C to gather the far-scattered
    photons, with few of them and with so many that their lists fill up."""
    import torch
    from marx_gb300._native import DevicePhotons, Engine, MODE_FUSED, MODE_WAVEFRONT
    w = W.plain_scatter()
    for k in range(4):
        w.cfg.scat_p[k] *= scat
        w.cfg.scat_h[k] *= scat
    eng, out = Engine(w.cfg), []
    ph = w.photons(3_000_001, seed=12)
    for mode in (MODE_FUSED, MODE_WAVEFRONT):
        d = DevicePhotons.from_host(ph)
        eng.set_mode(mode)
        eng.trace(d, seed=13)
        out.append(d)
    for c in ("x", "p", "flags", "mirror_shell", "ccd_num", "y_pixel", "z_pixel"):
        assert torch.equal(getattr(out[0], c), getattr(out[1], c)), c
