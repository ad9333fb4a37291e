"""Gas blocks whose pencils end in outflow, reflecting or mixed rules: the
one-launch sweep (k_sweep_open) against the oracle, bit for bit, guard cells
included -- short pencils, the longest the CTA holds and one cell more (the
stage path), every rule on either side, dust beside the gas, guard cells that
the caller filled differently (the first sweep then reads those, as the
oracle does), steps replayed from a graph and redone steps."""
import numpy as np
import pytest

from helpers import assert_bitexact, random_state, setup_for
from piernik_b200._lib import PK_RK2_1
from piernik_b200.config import BND_OUT, BND_PER, BND_REF
from piernik_b200.sim import Simulation

pytestmark = pytest.mark.gpu

O, P, R = (BND_OUT, BND_OUT), (BND_PER, BND_PER), (BND_REF, BND_REF)
OR, RO = (BND_OUT, BND_REF), (BND_REF, BND_OUT)


def _check(sim, ob, what):
    gu, _, _ = sim.download()
    assert_bitexact(gu, ob.u, what)
    st = sim.time_state
    assert (st.t, st.dt, st.nstep) == (ob.state.t, ob.state.dt, ob.state.nstep), what


@pytest.mark.parametrize("n,bnd", [((5, 4, 6), (O, R, OR)), ((33, 20, 17), (R, O, P)), ((252, 6, 5), (RO, O, R)),
                                   ((253, 6, 5), (RO, O, R)), ((6, 300, 5), (R, OR, O)), ((7, 5, 252), (P, R, RO)),
                                   ((40, 30, 1), (O, RO, P)), ((64, 1, 1), (R, P, P))])
@pytest.mark.parametrize("lim", ["vanleer", "superbee"])
def test_open_blocks_bitexact(gpu_lib, oracle_lib, n, bnd, lim):
    setup = setup_for("hd", n=n, lim=lim, bnd=bnd)
    u, _, _ = random_state(setup, seed=2)
    sim = Simulation(setup)
    sim.upload(u)
    ob = oracle_lib.OracleBlock(setup, u, None, None)
    for k in range(2):                     # the first from the caller's (periodic) guard cells
        sim.run(1)
        ob.run(1)
        _check(sim, ob, f"{n} {bnd} step {k}")
    sim.run(2)
    ob.run(2)
    _check(sim, ob, f"{n} {bnd} steps 3, 4")
    sim.close()


@pytest.mark.parametrize("how", ["graph", "redo", "dust", "single sweeps"])
def test_open_blocks_options(gpu_lib, oracle_lib, how):
    setup = setup_for("hd", n=(24, 18, 270 if how == "graph" else 14), lim="minmod", bnd=(OR, R, O))
    if how == "redo":
        setup = setup.replace(cflcontrol="redo", cfl=0.9)
    if how == "dust":
        setup = setup.replace(fluids=[("neu", 1.4), ("dst", -1.0)])
    u, _, _ = random_state(setup, seed=4)
    sim = Simulation(setup)
    start = sim.time_state
    sim.upload(u)
    ob = oracle_lib.OracleBlock(setup, u, None, None)
    if how == "graph":
        sim.use_graph()
    if how == "single sweeps":
        for d, drop_in in ((1, False), (3, False), (2, True), (2, False), (1, False)):
            if drop_in:                    # a stage of the drop-in entry point leaves guard cells of its own
                sim.solve_cg(d, PK_RK2_1, 0.001)
                ob.solve_cg(d - 1, 1, 0.001, 0.0)
            else:
                sim.sweep(d, 0.002)
                ob.sweep(d - 1, 0.002, 0.0)
        gu, _, _ = sim.download()
        assert_bitexact(gu, ob.u, how)
    else:
        sim.run(3)
        ob.run(3)
        _check(sim, ob, how)
        sim.upload(u)                      # the caller's guard cells again, in the middle of a run
        ob2 = oracle_lib.OracleBlock(setup, u, None, None)
        sim.time_state = start
        sim.run(2)
        ob2.run(2)
        gu, _, _ = sim.download()
        assert_bitexact(gu, ob2.u, how + " after a new upload")
    sim.close()
