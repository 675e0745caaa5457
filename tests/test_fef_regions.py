"""An FEF region of a single energy has nothing to interpolate between: the
configuration is refused (no GPU needed), as one with two energies is not."""
import os

import pytest

from helpers import GOLDEN
from marx_gb300 import workloads as W
from marx_gb300.caldb.pack import DEFAULT_PACK, pack_with_fef, read_pack, write_pack


@pytest.mark.parametrize("energies,ok", [(1, False), (2, True)])
def test_regions_of_one_energy_are_refused(tmp_path, energies, ok):
    from marx_gb300._native import validate_config
    pack = str(tmp_path / "fef.mxpack")
    pack_with_fef(DEFAULT_PACK, os.path.join(GOLDEN, "acis_fef_synthetic.fits"), pack)
    S = read_pack(pack)
    rows = S["acis/fef/rows"]
    first = [k for k in range(len(rows)) if k == 0 or rows[k, 5] != rows[k - 1, 5]]   # of each region
    keep = sorted(f + j for f in first for j in range(energies))
    S["acis/fef/rows"], S["acis/fef/vals"] = rows[keep], S["acis/fef/vals"][keep]
    write_pack(pack, S)
    got = validate_config(W.ALL["plain_scatter"](parity=True).cfg, pack=pack)
    assert (got is None) if ok else ("more than one energy" in (got or ""))
