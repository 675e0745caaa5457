"""Weighted rays at the edges of their kernels: ragged and tiny ray counts,
large tilts and decenters (rays that leave the Newton intersection for the
closed form), images smaller than the shared window and off the image
centre, against the CPU restatement and numpy.

Tolerances: a ray's focal-plane position is good to 1e-9 mm and its weight to
1e-12 (the bounds of the oracle comparison at the workload's own geometry;
tilts leave the magnitudes as they are); image pixels to 1e-9 of the largest
(a tap is a single-precision value, the same on both sides but where the last
bits of a position decide its rounding)."""
import numpy as np
import pytest

from marx_gb300.diff import DiffImage, diff_mirror_config, diff_workload, NPARAM, RECORD, REPLAY, FRESH

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine(cuda):
    from marx_gb300._native import Engine
    return Engine(diff_mirror_config(ideal=False))


def _theta(scale):
    t = np.random.default_rng(11).normal(0.0, scale, NPARAM)
    t[16:] = np.clip(t[16:], -120.0, 120.0)
    return t


@pytest.mark.parametrize("scale", [0.0, 30.0, 600.0])
@pytest.mark.parametrize("n", [1, 31, 33, 255, 20_011])
def test_rays_image_and_moments_match_oracle(engine, n, scale):
    from oracle.bindings import Oracle
    theta = _theta(scale)
    w = diff_workload(n_rays=n)
    cfg = w.cfg.copy()
    cfg.nx, cfg.ny = 16, 80          # narrower than the 64 x 64 window, and taller
    cfg.center_z += 20 * cfg.pitch   # rays across the window's edge
    d = DiffImage(engine, cfg)
    yzw = d.rays(theta, FRESH).cpu().numpy()
    oy, oimg = Oracle(diff_mirror_config(ideal=False)).weighted(cfg, theta)
    hit = yzw[2] > 0
    assert np.array_equal(hit, oy[2] > 0)
    if hit.any():
        assert np.abs(yzw[:2, hit] - oy[:2, hit]).max() <= 1e-9
        assert np.abs(yzw[2, hit] / oy[2, hit] - 1.0).max() <= 1e-12
    img = d.forward(theta, FRESH).cpu().numpy()
    assert np.abs(img - oimg).max() <= 1e-9 * max(oimg.max(), 1e-300)
    m = d.moments(theta, FRESH)
    assert m[3] == hit.sum()
    want = [yzw[2, hit].sum(), (yzw[2, hit] * yzw[0, hit]).sum(), (yzw[2, hit] * yzw[1, hit]).sum()]
    size = [np.abs(yzw[2, hit]).sum(), np.abs(yzw[2, hit] * yzw[0, hit]).sum(), np.abs(yzw[2, hit] * yzw[1, hit]).sum()]
    for a, b, s in zip(m[:3], want, size):
        assert abs(a - b) <= 1e-12 * s + 1e-300
    d.close()


@pytest.mark.parametrize("n", [33, 20_011])
def test_replay_follows_the_recorded_rays(engine, n):
    w = diff_workload(n_rays=n)
    d = DiffImage.centred(engine, w.cfg)
    a, b = _theta(0.5), _theta(30.0)
    img = d.forward(a, RECORD)
    assert bool((d.forward(a, REPLAY) == img).all())
    rec, moved, fresh = (d.rays(t, m).cpu().numpy() for t, m in ((a, REPLAY), (b, REPLAY), (b, FRESH)))
    assert np.array_equal(rec[2] > 0, moved[2] > 0)   # the same rays, wherever the mirrors are
    both = (moved[2] > 0) & (fresh[2] > 0)
    assert both.sum() >= n // 8
    assert np.abs(moved[:2, both] - fresh[:2, both]).max() <= 1e-9
    d.close()


@pytest.mark.parametrize("nx,ny", [(16, 16), (31, 33), (257, 250)])
def test_mse(engine, nx, ny):
    import torch
    w = diff_workload(n_rays=100)
    cfg = w.cfg.copy()
    cfg.nx, cfg.ny = nx, ny
    d = DiffImage(engine, cfg)
    g = torch.Generator().manual_seed(3)
    a, b = (torch.rand((ny, nx), generator=g, dtype=torch.float64) for _ in range(2))
    loss, dl = d.mse(a.cuda(), b.cuda())
    r = (a - b).numpy()
    assert float(loss) == pytest.approx(float((r * r).mean()), rel=1e-13)
    np.testing.assert_allclose(dl.cpu().numpy().reshape(ny, nx), 2.0 * r / (nx * ny), rtol=4e-16, atol=0)
    d.close()


@pytest.mark.parametrize("ideal", [False, True])
@pytest.mark.parametrize("n,scale", [(1, 0.5), (33, 0.5), (130, 30.0), (20_011, 0.5), (20_011, 30.0)])
def test_adjoint_matches_central_differences(cuda, n, scale, ideal):
    """The adjoint of a linear function of the image, sum dl image, whose
    gradient keeps one sign over rays and taps (dl rises along both axes).
    Tolerance: the derivatives are sums of single-precision terms (1e-5 of
    their size at worst); the taps' rounding (2^-24) over the 4e-3 pixels of
    a step of 2e-3 arcsec gives the differences 3e-5, and the third order
    they leave out 1e-5: 1e-3 of the gradient's norm leaves room for the
    tilts' smaller steps."""
    import torch
    from marx_gb300._native import Engine
    theta = _theta(scale)
    eng = Engine(diff_mirror_config(ideal=ideal))
    centred = DiffImage.centred(eng, diff_workload(n_rays=20_011).cfg, theta)   # one ray alone may miss
    cfg = centred.cfg.copy()
    cfg.n_rays = n
    cfg.nx, cfg.ny = 40, 80
    cfg.center_z += 25 * cfg.pitch   # rays across the window's edge
    d = DiffImage(eng, cfg)
    row, col = np.mgrid[0:cfg.ny, 0:cfg.nx]
    dl = torch.from_numpy(0.3 + 0.01 * col + 0.007 * row + 2e-4 * col * row).cuda()
    d.forward(theta, RECORD)
    g = d.adjoint(theta, dl)
    h, fd = 2e-3, np.empty(NPARAM)
    for k in range(NPARAM):
        v = []
        for sign in (1.0, -1.0):
            t = theta.copy()
            t[k] += sign * h
            v.append(float((d.forward(t, REPLAY) * dl).sum()))
        fd[k] = (v[0] - v[1]) / (2 * h)
    assert np.linalg.norm(g - fd) <= 1e-3 * np.linalg.norm(fd), (g, fd)
    assert np.array_equal(g, d.adjoint(theta, dl))
    d.close()
    centred.close()
