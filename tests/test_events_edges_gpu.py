"""The event pass where its branches meet: pixels on sub-pixel thirds, sky
offsets and dithers on both sides of the series' range, rolls beyond a turn,
detector motion, and list lengths at the edges of the tiles, against the CPU
oracle with the tolerances of test_events_gpu."""
import numpy as np
import pytest

from marx_gb300 import events as E
from marx_gb300.caldb.pack import DEFAULT_PACK, read_pack
from oracle.event_coords import PIXADJ, event_coords as oracle_coords, subpix_tables

from test_events import load_case
from test_events_gpu import check_against_oracle, engine_for, synthetic_events

pytestmark = pytest.mark.gpu


def compare(ev, U, mode, det="acis_i"):
    z, det, params, _ = load_case(det)
    p = E.params(focal_length=params["focal_length"], det_offset=params["det_offset"], roll_nom=params["roll_nom"],
                 frame_time=params["frame_time"], dithered=True, pixel_adjust=mode)
    g = E.event_coords_host(engine_for(det), p, dict(ev, uniforms=U))
    params["pixel_adjust"] = PIXADJ[mode]
    with np.errstate(invalid="ignore"):
        o = oracle_coords(det, z["geom"], z["tdet"], z["fp"], params, ev, U, subpix_tables(read_pack(DEFAULT_PACK)))
    check_against_oracle(g, o, ev, f"{mode} {len(U[0])}")


# tile edges of a short list (256-event tiles), and where tiles of four
# rounds take over (8 blocks per SM x 4 x 256 events, 152 SMs)
@pytest.mark.parametrize("n", [1, 31, 32, 255, 256, 257, 152 * 8 * 4 * 256 - 1, 152 * 8 * 4 * 256 + 1])
def test_list_lengths(cuda, n):
    z, _, params, _ = load_case("acis_i")
    ev, U = synthetic_events(n, z["geom"], 11, params["frame_time"], 70)
    compare(ev, U, "NONE")


@pytest.mark.parametrize("mode", ["EDSER", "EXACT", "RANDOMIZE"])
def test_branches_meet(cuda, mode):
    z, _, params, _ = load_case("acis_i")
    n, f = 40_000, np.float32
    ev, U = synthetic_events(n, z["geom"], 12, params["frame_time"], 3)
    r = np.random.default_rng(13)
    # fractions at, just below and just above 0, 1/3, 2/3 and 1
    third = np.array([0, 1, 2, 3], f) / f(3)
    base = r.integers(0, 1024, n).astype(f)
    for c in ("xpixel", "ypixel"):
        v = (base + third[r.integers(0, 4, n)]).astype(f)
        ev[c] = np.where(r.random(n) < 0.5, np.nextafter(v, f(-1)), v).astype(f)
    far = slice(0, n // 4)            # up to 0.07 rad off: both sides of the series' 0.03
    ev["xpixel"][far] = r.uniform(-3e4, 3e4, n // 4)
    q = slice(n // 4, n // 2)         # dithers around 1e-4 rad, and none
    ev["sky_ra"][q] = r.choice(np.array([0, 9.99e-5, 1.01e-4, -3e-3, 1e-12], f), n // 4)
    ev["sky_dec"][q] = r.choice(np.array([0, -9.99e-5, 1.01e-4, 2e-3], f), n // 4)
    q = slice(n // 2, 3 * n // 4)     # rolls over more than a turn
    ev["sky_roll"][q] = r.uniform(-9, 9, n // 4)
    q = slice(3 * n // 4, n)          # detector motion and rotation
    ev["det_dy"][q] = r.normal(0, 0.02, n // 4)
    ev["det_dz"][q] = r.normal(0, 0.02, n // 4)
    ev["b_energy"][::7] = r.choice(np.array([0.0, 0.1, 20.0], f), len(ev["b_energy"][::7]))   # outside the tables
    compare(ev, U, mode)
    ev["det_theta"][q] = r.normal(0, 2e-5, n // 4)
    compare(ev, U, mode)
