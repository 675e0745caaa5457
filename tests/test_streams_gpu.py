"""Calls of one context on several streams: they share the context's survivor
queues, its frame scan and its table of the source's spectrum, and give what
the same calls give with a wait after each.  No tolerance: every column is
equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
COLUMNS = ("x", "p", "flags", "mirror_shell", "order", "ccd_num", "y_pixel", "z_pixel")


def _wait():
    import torch
    torch.cuda.synchronize()


@pytest.mark.parametrize("streams", [1, 3])
def test_traces_take_turns_at_the_queues(cuda, streams):
    """Lists short enough for one pass and too long for the fused kernel."""
    import torch
    from marx_gb300 import workloads as W
    from marx_gb300._native import DevicePhotons, Engine
    w = W.plain_hetg()
    eng = Engine(w.cfg)
    lists = [w.photons(n, seed=n) for n in (150_001, 98_000, 200_000, 120_033, 99_999, 260_000)]
    out, side = [], [torch.cuda.Stream() for _ in range(streams)]
    for apart in (True, False):
        d = [DevicePhotons.from_host(q) for q in lists]
        _wait()
        for k, q in enumerate(d):
            eng.trace(q, stages=w.stages, seed=k, stream=side[k % streams])
            if apart:
                _wait()
        _wait()
        out.append(d)
    for a, b in zip(*out):
        for c in COLUMNS:
            assert torch.equal(getattr(a, c), getattr(b, c)), c


@pytest.mark.parametrize("streams", [1, 2])
@pytest.mark.parametrize("kind", ["spectrum", "image"])
def test_sources_take_turns_at_the_table(cuda, kind, streams):
    """Tables of one length, then a longer one: each source draws from its own."""
    import torch
    from marx_gb300 import batched as B
    from marx_gb300._native import DevicePhotons, Engine
    eng = Engine(B.batched_config())
    n, p, r = 3_000_000, np.array([-1.0, 0.0, 0.0]), np.random.default_rng(4)
    sources = []
    for k in range(5):
        m = 300 if k < 4 else 3000
        if kind == "spectrum":
            spec = (np.linspace(0.3 + 0.1 * k, 2.0 + k, m), r.random(m))
            sources.append(B.make_source(p, "POINT", (), spectrum=spec, num_photons=n))
        else:
            sources.append(B.make_source(p, "IMAGE", (1e-4, 1e-4), image=r.random((10, m // 10)).astype(np.float32),
                                         num_photons=n))
    side = [torch.cuda.Stream() for _ in range(streams)]
    out = []
    for apart in (True, False):
        d = [DevicePhotons(n) for _ in sources]
        _wait()
        for k, (s, q) in enumerate(zip(sources, d)):
            B.generate_source(eng, s, 0, k, q, stream=side[k % streams])
            if apart:
                _wait()
        _wait()
        out.append(d)
    for a, b in zip(*out):
        for c in ("energy", "p"):
            assert torch.equal(getattr(a, c), getattr(b, c)), c


def test_event_passes_take_turns_at_the_frame_scan(cuda):
    import torch
    from marx_gb300 import events as E
    from test_events import load_case
    from test_events_gpu import engine_for, synthetic_events
    z, det, params, _ = load_case("acis_i")
    eng = engine_for(det)
    p = E.params(focal_length=params["focal_length"], det_offset=params["det_offset"], roll_nom=params["roll_nom"],
                 frame_time=params["frame_time"], dithered=True, pixel_adjust="NONE")
    sets = []
    for k, n in enumerate((1_500_000, 3_000, 900_001, 400_000)):
        ev, _ = synthetic_events(n, z["geom"], 20 + k, params["frame_time"], 30)
        sets.append((n, {c: torch.from_numpy(np.ascontiguousarray(v, dtype=E.INPUTS[c][1])).cuda()
                         for c, v in ev.items() if v is not None}))
    side = [torch.cuda.Stream() for _ in range(3)]
    out = []
    for apart in (True, False):
        _wait()
        got = []
        for k, (n, ev) in enumerate(sets * 2):
            with torch.cuda.stream(side[k % 3]):   # its outputs belong to that stream
                got.append(E.event_coords(eng, p, ev, n, seed=k))
            if apart:
                _wait()
        _wait()
        out.append(got)
    for a, b in zip(*out):
        for c, v in a.items():
            assert torch.equal(v.view(torch.uint8), b[c].view(torch.uint8)), c
