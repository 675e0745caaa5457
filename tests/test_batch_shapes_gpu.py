"""The launch shapes that mx_batch_set_params takes: up to 24 warps per SM (768
threads), however many of a shape's blocks the kernel's registers and shared
memory leave room for, and no more; and the most sources a batch may have.  A
batch gives the same photons in each."""
import pytest

from marx_gb300 import batched as B
from helpers import assert_parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsrc", [3, 380])
@pytest.mark.parametrize("block", [32, 64, 96, 128, 160, 192, 224, 256])
def test_shapes_of_24_warps_per_sm(cuda, nsrc, block):
    import torch
    from marx_gb300._native import Engine
    b = B.Batch(Engine(B.batched_config()), B.batched_sources(nsrc=nsrc, seed=5, nmin=20, nmax=300))
    b.run(seed=13)
    torch.cuda.synchronize()
    ref = b.to_host()
    # 380 sources take 68 KB of shared memory a block with the tables: three blocks
    most = 768 // block if nsrc == 3 else min(3, 768 // block)
    for per_sm in (1, most):
        b.set_params(block, 64, per_sm)
        assert b.params() == {"block": block, "tile": 64, "blocks_per_sm": per_sm}
        b.run(seed=13)
        torch.cuda.synchronize()
        assert_parity(b.to_host(), ref, f"{nsrc} sources, block {block}, {per_sm} per SM")
    with pytest.raises(RuntimeError, match="more blocks per SM than fit"):
        b.set_params(block, 64, most + 1)


def test_most_sources(cuda):
    """1252 sources are the most that one block's shared memory takes with
    their offsets; the last ones' photons come out as from a short batch."""
    import torch
    from marx_gb300._native import Engine
    eng = Engine(B.batched_config())
    b = B.Batch(eng, B.batched_sources(nsrc=1252, seed=5, nmin=20, nmax=300))
    b.run(seed=13)
    torch.cuda.synchronize()
    ref = b.to_host()
    b.run_sequential(seed=13)
    torch.cuda.synchronize()
    assert_parity(ref, b.to_host(), "1252 sources")
    with pytest.raises(RuntimeError, match="cannot be resident"):
        B.Batch(eng, B.batched_sources(nsrc=1253, seed=5, nmin=20, nmax=300))
