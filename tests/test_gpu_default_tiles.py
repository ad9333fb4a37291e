"""Sweeps in the tiles that the library picks by size when no one tuned them
(default_tile in pk_launch.cuh), against the oracle bit for bit: extents on
either side of each of the rule's lines -- staged whole pencils, whole pencils
in one CTA, chunks along x and across it, blocks too small for the rule --
with even and odd extents along x (the staged kernel needs even ones)."""
import numpy as np
import pytest

from helpers import assert_bitexact, random_state, setup_for
from piernik_b200.sim import Simulation

pytestmark = pytest.mark.gpu

SIZES = [(64, 64, 64),        # staged along every direction
         (63, 64, 65),        # odd x: whole pencils along x, y; chunks along z
         (128, 40, 36),       # too few pencils for the staged kernel
         (258, 16, 12),       # x longer than a CTA: chunks
         (12, 16, 258),       # the same along z, staged along x refused by its size
         (8, 70, 64), (32, 32, 32), (31, 32, 32),
         (256, 200, 1), (300, 130, 1)]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("phys", ["hd", "mhd"])
def test_untuned_sweeps_bitexact(gpu_lib, oracle_lib, phys, n):
    setup = setup_for(phys, n=n, lim="moncen")
    u, b, psi = random_state(setup, seed=3)
    sim = Simulation(setup)
    sim.upload(u, b, psi)
    ob = oracle_lib.OracleBlock(setup, u, b, psi)
    sim.run(1)
    ob.run(1)
    gu, gb, gp = sim.download()
    assert_bitexact(gu, ob.u, f"u {phys} {n}")
    if setup.magnetic:
        assert_bitexact(gb, ob.b, f"b {n}")
        assert_bitexact(gp, ob.psi, f"psi {n}")
    sim.close()


@pytest.mark.parametrize("seg", [40, 130])
def test_untuned_stacked_instances_equal_lone_runs(gpu_lib, seg):
    """Stacked instances sweep z segment by segment (40 cells: six pencils a
    CTA, 130: three); each must equal the same problem run alone."""
    one = setup_for("mhd", n=(36, 34, seg), lim="vanleer")
    states = [random_state(one, seed=s) for s in (1, 2)]
    g = one.guards[2]
    both = one.replace(n=(36, 34, 2 * seg), xmax=(one.xmax[0], one.xmax[1], 2 * one.xmax[2]))

    def stack(i):
        core = [s[i][g:-g] for s in states]
        return np.concatenate([core[1][-g:], *core, core[0][:g]])

    sim = Simulation(both)
    sim.upload(*(np.ascontiguousarray(stack(i)) for i in range(3)))
    sim.set_instances(2)
    sim.run(2)
    got = sim.download()
    sim.close()
    for k, st in enumerate(states):
        lone = Simulation(one)
        lone.upload(*st)
        lone.run(2)
        want = lone.download()
        lone.close()
        for a, w, name in zip(got, want, ("u", "b", "psi")):
            cut = (slice(g + k * seg, g + (k + 1) * seg), slice(4, -4), slice(4, -4))
            assert_bitexact(np.ascontiguousarray(a[cut]), np.ascontiguousarray(w[g:-g, 4:-4, 4:-4]), f"{name} of instance {k}")
