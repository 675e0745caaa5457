"""The batch kernel's work lists at their edges: batches of one photon to some
hundred thousand, launch shapes in which a warp keeps a list of far-scattered
photons for later (a queue of three groups or more per warp) and in which it
does not, tiles larger than a phase has work.  Equal to the sources traced one
by one, as the batch at its default shape is."""
import pytest

from marx_gb300 import batched as B
from helpers import assert_parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsrc,nmin,nmax", [(1, 1, 1), (3, 31, 33), (7, 2000, 9000), (40, 500, 60_000)])
@pytest.mark.parametrize("block,tile,per_sm", [(256, 256, 2), (32, 32, 1), (96, 1024, 1)])
def test_batch_equals_sources_one_by_one(cuda, nsrc, nmin, nmax, block, tile, per_sm):
    import torch
    from marx_gb300._native import Engine
    b = B.Batch(Engine(B.batched_config()), B.batched_sources(nsrc=nsrc, seed=21, nmin=nmin, nmax=nmax))
    b.set_params(block, tile, per_sm)
    b.run(seed=13)
    torch.cuda.synchronize()
    one = b.to_host()
    b.run_sequential(seed=13)
    torch.cuda.synchronize()
    assert_parity(one, b.to_host(), f"{nsrc} sources, block {block}, tile {tile}")
