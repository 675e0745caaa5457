"""Photons whose directions are not of unit length to the last bits (widened
from single precision, or off by parts in 1e10): the mirror's closed forms,
which take a direction for a unit vector, decide where they meet it, so that
they arrive where the CPU restatement of the reference puts them, within the
parity contract's 1e-9 mm and 1e-12.  In a list of them among unit vectors,
in each kind of kernel, and from a POINT source of a batch."""
import os

import numpy as np
import pytest

from marx_gb300 import batched as B
from marx_gb300 import workloads as W
from marx_gb300.photons import PhotonList

from helpers import assert_parity

pytestmark = pytest.mark.gpu


def _photons(n, change):
    r = np.random.default_rng(31)
    p = W.offaxis_directions(r.uniform(0, 8, n) * W.ARCMIN, r.uniform(0, 2 * np.pi, n))
    return PhotonList.from_inputs(r.uniform(0.3, 8, n), np.ascontiguousarray(change(p, r)), r.uniform(0, 1e4, n))


CHANGES = {"widened": lambda p, r: p.astype(np.float32).astype(np.float64),
           "longer": lambda p, r: p * (1 + 1e-10),
           "every other": lambda p, r: p * np.where(r.random(p.shape[1]) < 0.5, 1.0, 1 - 3e-8)}


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("name", ["plain_onaxis", "plain_scatter"])
@pytest.mark.parametrize("change", sorted(CHANGES))
def test_positions_as_the_reference_has_them(cuda, name, change, mode):
    from marx_gb300._native import Engine
    from oracle.bindings import Oracle
    w = W.ALL[name]()
    q = _photons(50_000, CHANGES[change])
    o = q.copy()
    eng = Engine(w.cfg)
    eng.set_mode(mode)
    eng.trace_host(q, stages=w.stages, seed=3)
    Oracle(w.cfg).trace(o, stages=w.stages, seed=3, threads=os.cpu_count() or 1)
    for c in ("flags", "mirror_shell", "ccd_num"):
        np.testing.assert_array_equal(getattr(q, c), getattr(o, c), err_msg=c)
    good = q.good()
    assert good.sum() > 1000
    assert np.max(np.abs(q.x - o.x)[:, good]) < 1e-9
    assert np.max(np.abs(q.p - o.p)[:, good]) < 1e-12


def test_batch_of_widened_sources(cuda):
    """The photons of a batch and of its sources traced one by one, and those
    of the source's own list on the CPU."""
    import torch
    from marx_gb300._native import Engine
    from oracle.bindings import Oracle
    cfg = B.batched_config()
    src = B.batched_sources(nsrc=5, seed=3, nmin=3000, nmax=9000)
    for s in src:
        s.p[:] = [float(np.float32(v)) for v in s.p]
    b = B.Batch(Engine(cfg), src)
    b.run(seed=4)
    torch.cuda.synchronize()
    one = b.to_host()
    b.run_sequential(seed=4)
    torch.cuda.synchronize()
    assert_parity(one, b.to_host(), "one by one")
    start = b.source_start()
    k = next(k for k in range(5) if src[k].grating == 0 and src[k].detector == B.DETECTOR["ACIS-I"])
    n, at = start[k + 1] - start[k], slice(start[k], start[k + 1])
    o = PhotonList.from_inputs(one.energy[at].copy(), np.repeat(np.array(src[k].p[:])[:, None], n, axis=1), np.zeros(n))
    o.tag[:] = np.arange(start[k], start[k + 1], dtype=np.uint32)
    cfg.grating, cfg.detector = 0, B.DETECTOR["ACIS-I"]
    Oracle(cfg).trace(o, seed=4, threads=os.cpu_count() or 1)
    np.testing.assert_array_equal(one.flags[at], o.flags)
    good = (o.flags & 0xFF) == 0
    assert good.sum() > 200
    assert np.max(np.abs(one.x[:, at] - o.x)[:, good]) < 1e-9
