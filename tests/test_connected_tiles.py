"""Tiles of a connected block's fused sweep (halo read from the guard cells)
that end beyond the pencil: the last chunk of a pencil longer than the batched
tile (56 cells), or of any pencil swept in chunks.

On the CPU: no thread of any tile may read outside the pencil with its guard
cells (fused_tile's positions and its active condition, for the tiles that
build_batch and the untuned single block make), every owned cell's four
neighbours on either side are read, and no cell of the tile is updated from
one that the tile does not hold (the kernels' own role functions, built for the
host).  On the GPU: a domain cut so must equal the same domain held as one
block, also with fewer than four guard layers, where connected blocks are swept
stage by stage, and raise the status that the one block raises: no step is
redone for cells that nobody stores."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from helpers import assert_bitexact, random_state, setup_for
from test_gpu_blocks import exact_dl, interior_of, run_tiled, tiles, window
from piernik_b200.sim import Simulation

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "piernik_b200", "csrc")


def _roles_lib():
    src, out = os.path.join(HERE, "native", "roles_harness.cu"), os.path.join(HERE, "native", "libroles_harness.so")
    deps = [src] + [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cuh")]
    if not os.path.exists(out) or os.path.getmtime(out) < max(os.path.getmtime(d) for d in deps):
        subprocess.check_call(["nvcc", "-std=c++17", "--fmad=false", "-Xcompiler", "-fPIC,-O2,-ffp-contract=off",
                               "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", out, src])
    return C.CDLL(out)


@pytest.mark.parametrize("wrap", [0, 1])
def test_no_role_needs_a_cell_the_tile_does_not_hold(wrap):
    """Both stages of every tile, as rk_stage runs them: a slope needs three
    cells' primitives, a flux two slopes, an update two fluxes, the second
    stage's primitives the first's update."""
    f = _roles_lib().fused_tile_roles
    for n in (4, 40, 56, 57, 60, 64, 72, 100, 113, 300):
        for L in (24, 56, 64):
            L = min(L, n)
            T = L + 8
            for c0 in range(0, n, L):
                out = (C.c_ubyte * (2 * T))()
                end = f(T, wrap, 0, c0, n, out)
                assert end == (T if wrap else min(T, n + 8 - c0))
                bits = np.array(out, dtype=np.uint8).reshape(2, T)
                state = np.arange(T) < end                      # the cells that are loaded
                for st in range(2):
                    q, slope, flux, upd = ((bits[st] >> k) & 1 == 1 for k in range(4))
                    what = f"n {n} L {L} c0 {c0} stage {st}"
                    assert not (q & ~state).any(), what
                    left, right = (lambda a: np.r_[False, a[:-1]]), (lambda a: np.r_[a[1:], False])
                    assert not (slope & ~(left(q) & q & right(q))).any(), what
                    assert not (flux & ~(slope & right(slope))).any(), what
                    assert not (upd & ~(left(flux) & flux)).any(), what
                    state = upd
                own = slice(4, 4 + min(L, n - c0))
                assert state[own].all() and own.stop - own.start > 0


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


@pytest.mark.gpu
@pytest.mark.parametrize("phys", ["hd", "mhd"])
@pytest.mark.parametrize("n,cuts", [((64, 12, 16), ([64], [12], [8, 8])), ((12, 100, 16), ([12], [100], [8, 8])),
                                    ((12, 16, 128), ([12], [8, 8], [113, 15]))])
def test_long_blocks_redo_no_step_for_cells_nobody_stores(gpu_lib, phys, n, cuts):
    """cflcontrol = redo repeats a step whose status says negative: the tiled
    domain must walk the one block's dt sequence, and raise nothing, whatever the
    shared memory held before (here: the states of a violent flow of no mean
    velocity in blocks of the same shape, swept just before on another handle)."""
    full = exact_dl(setup_for(phys, n=n, lim="moncen", cflcontrol="redo", cfl_max=0.9))
    state = random_state(full, seed=11)
    rng = np.random.default_rng(5)
    wild = [x.copy() if x is not None else None for x in random_state(full, seed=12)]
    wild[0][..., 1:4] = rng.choice([-1e4, 1e4], wild[0].shape[:3] + (3,)) * wild[0][..., :1]
    wild[0][..., 4] += 1.5e8 * wild[0][..., 0]

    def tiled(st):
        sim = None
        for bn, off in tiles(*cuts):
            s = full.replace(n=bn, xmin=tuple(full.xmin[d] + off[d] * full.dl[d] for d in range(3)),
                             xmax=tuple(full.xmin[d] + (off[d] + bn[d]) * full.dl[d] for d in range(3)))
            if sim is None:
                sim, bid = Simulation(s), 0
                sim.set_domain(full.n, (True, True, True))
            else:
                bid = sim.add_block(s)
            sim.place_block(bid, off)
            sim.upload(*(window(full, x, bn, off) for x in st), block=bid)
        sim.update_boundaries()
        return sim

    one, sim, other = Simulation(full), tiled(state), tiled(wild)
    one.upload(*state)
    for cdim in (1, 2, 3, 3, 2, 1):
        other.sweep(cdim, 1e-9, 1.0)
        other.sync()
        for x in (one, sim):
            x.sweep(cdim, 1e-3, 1.0)
        assert sim.status() == one.status() == 0, cdim
    for _ in range(4):
        other.sweep(1, 1e-9, 1.0)
        other.sync()
        for x in (one, sim):
            x.run(1)
        a, c = one.time_state, sim.time_state
        assert (a.t, a.dt, a.redone, a.repeat_step) == (c.t, c.dt, c.redone, c.repeat_step)
    for x in (one, sim, other):
        x.close()
