"""Device traces captured into a CUDA graph (the wavefront's phases are
launched with programmatic stream serialisation, a list of 2^18 photons or
more in two halves on two streams): replays equal the direct trace byte for
byte, with the line between the fused and the wavefront kernels crossed."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,n", [("plain_scatter", 97_280), ("plain_scatter", 97_281), ("plain_hetg", 80_000),
                                    ("plain_hetg", 150_001), ("letg_hrcs", 300_001)])
def test_captured_trace_equals_direct(cuda, name, n):
    import torch
    from marx_gb300 import workloads as W
    from marx_gb300._native import DevicePhotons, Engine
    w = W.ALL[name]()
    eng = Engine(w.cfg)
    d = DevicePhotons.from_host(w.photons(n))
    p0 = d.p.clone()
    keep = {}
    for mode in (1, 2, 0):     # fused, wavefront, the choice between them: the same results
        eng.set_mode(mode)
        d.p.copy_(p0)
        d.flags.zero_()
        eng.trace(d, stages=w.stages, seed=3)
        torch.cuda.synchronize()
        now = {k: getattr(d, k).clone() for k in ("x", "p", "flags", "mirror_shell", "order", "ccd_num", "y_pixel")}
        for k, v in keep.items():
            assert torch.equal(v, now[k]), (mode, k)
        keep = now
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        eng.trace(d, stages=w.stages, seed=3)
    for _ in range(3):
        d.p.copy_(p0)
        d.flags.zero_()
        d.x.zero_()
        g.replay()
        torch.cuda.synchronize()
        for k, v in keep.items():
            assert torch.equal(v, getattr(d, k)), k
