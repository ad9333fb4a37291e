"""Tiles of a connected block's fused sweep (halo read from the guard cells)
that end beyond the pencil: the last chunk of a pencil longer than the batched
tile (56 cells), or of any pencil swept in chunks.

On the CPU: no thread of any tile may read outside the pencil with its guard
cells (fused_tile's positions and its active condition, for the tiles that
build_batch and the untuned single block make), and every owned cell's four
neighbours on either side are read.  On the GPU: a domain cut so must equal
the same domain held as one block, also with fewer than four guard layers,
where connected blocks are swept stage by stage."""
import numpy as np
import pytest

from helpers import assert_bitexact, random_state, setup_for
from test_gpu_blocks import exact_dl, interior_of, run_tiled, tiles
from piernik_b200.sim import Simulation


@pytest.mark.parametrize("n", [4, 40, 56, 57, 64, 72, 100, 113, 300])
@pytest.mark.parametrize("L", [24, 56, 64])
def test_no_tile_reads_past_the_guards(n, L):
    nb, L = 4, min(L, n)
    T = L + 8
    for c0 in range(0, n, L):
        s = [c0 - 4 + t for t in range(T) if c0 - 4 + t < n + 4]     # the active threads' positions
        assert min(s) + nb >= 0 and max(s) + nb < n + 2 * nb
        own = [x for t, x in enumerate(range(c0 - 4, c0 - 4 + T)) if 4 <= t < T - 4 and x < c0 + L and x < n]
        assert own == list(range(c0, min(c0 + L, n)))
        assert set(range(own[0] - 4, own[-1] + 5)) <= set(s)


def _equal_one_block(phys, n, cuts, **kw):
    full = exact_dl(setup_for(phys, n=n, lim="vanleer", **kw))
    state = random_state(full, seed=7)
    one = Simulation(full)
    one.upload(*state)
    one.run(2)
    ref = one.download()
    one.close()
    blocks = tiles(*cuts)
    got, _ = run_tiled(full, state, blocks, (True, True, True), 2)
    for (bn, off), arrs in zip(blocks, got):
        s = full.replace(n=bn)
        for a, r, name in zip(arrs, ref, ("u", "b", "psi")):
            if a is not None:
                assert_bitexact(interior_of(s, a, bn, (0, 0, 0)), interior_of(full, r, bn, off), f"block {off} {name}")


@pytest.mark.gpu
@pytest.mark.parametrize("phys", ["hd", "mhd"])
@pytest.mark.parametrize("n,cuts", [((96, 12, 16), ([64, 32], [12], [8, 8])), ((12, 90, 16), ([12], [66, 24], [16])),
                                    ((12, 16, 128), ([12], [8, 8], [113, 15])), ((100, 8, 8), ([100], [8], [8]))])
def test_long_blocks_equal_one_block(gpu_lib, phys, n, cuts):
    _equal_one_block(phys, n, cuts)


@pytest.mark.gpu
@pytest.mark.parametrize("phys", ["hd", "mhd"])
def test_narrow_guards_equal_one_block(gpu_lib, phys):
    _equal_one_block(phys, (24, 16, 12), ([8, 16], [16], [12]), nb=2)
