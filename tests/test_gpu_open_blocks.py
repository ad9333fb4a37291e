"""Gas blocks whose pencils end in outflow, reflecting or mixed rules: the
one-launch sweep (k_sweep_open) against the oracle, bit for bit, guard cells
included -- short pencils, the longest the CTA holds and one cell more (the
stage path), every rule on either side, dust beside the gas, guard cells that
the caller filled differently (the first sweep then reads those, as the
oracle does), steps replayed from a graph and redone steps.  The floors run over
the guard cells too, as the reference's do: where only one of those goes
negative the status must say so and a step be redone."""
import numpy as np
import pytest

from helpers import assert_bitexact, random_state, setup_for
from piernik_b200 import problems
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


def rough_state(setup, seed, mach):
    """Densities and pressures over two decades, velocities of either sign."""
    rng = np.random.default_rng(seed)
    u, _, _ = problems._empty(setup)
    shp, g = (setup.n[2], setup.n[1], setup.n[0]), setup.guards
    rho, p = 10 ** rng.uniform(-1, 1, shp), 10 ** rng.uniform(-1, 1, shp)
    v = rng.uniform(-mach, mach, shp + (3,))
    sl = tuple(slice(g[d], g[d] + setup.n[d]) for d in (2, 1, 0))
    problems._set_fluid(setup, u[sl], 0, rho, v[..., 0], v[..., 1], v[..., 2], p, None)
    return u


# seeds whose first sweep of a 6 x 4 x 5 reflecting box along the axis turns a guard
# cell negative and no interior one, in stage 1 or 2, found with the oracle
GUARD_ONLY = [("minmod", 6, 1, 2), ("minmod", 6, 14, 0), ("minmod", 6, 21, 0), ("minmod", 6, 27, 1),
              ("moncen", 6, 0, 1), ("moncen", 6, 49, 1), ("superbee", 3, 55, 0), ("vanleer", 6, 40, 2)]


@pytest.mark.parametrize("lim,mach,seed,axis", GUARD_ONLY + [("minmod", 1, 3, 0), ("moncen", 10, 4, 1)])
@pytest.mark.parametrize("bnd", [R, O, OR])
def test_floors_of_guard_cells_raise_the_status(gpu_lib, oracle_lib, lim, mach, seed, axis, bnd):
    setup = setup_for("hd", n=(6, 4, 5), lim=lim, bnd=(bnd,) * 3)
    ob = oracle_lib.OracleBlock(setup, rough_state(setup, seed, mach), None, None)
    ob.fill_guards()
    sim = Simulation(setup)
    sim.upload(ob.u)
    sim.update_boundaries()                # guard cells by the rules: the one-launch sweep
    dt, _ = ob.timestep_raw()
    for k in range(2):
        ob.blk.dn_negative = ob.blk.ei_negative = 0
        ob.sweep(axis, dt, 0.0)
        sim.sweep(axis + 1, dt)
        assert sim.status() == ob.blk.dn_negative + 2 * ob.blk.ei_negative, k
    gu, _, _ = sim.download()
    assert_bitexact(gu, ob.u, f"{lim} {seed}")
    sim.close()


@pytest.mark.parametrize("lim,mach,seed,axis", GUARD_ONLY)
def test_a_negative_guard_cell_redoes_the_step(gpu_lib, oracle_lib, lim, mach, seed, axis):
    """Sweeps along one axis only, so that the step is redone for nothing else."""
    setup = setup_for("hd", n=(6, 4, 5), lim=lim, bnd=(R,) * 3, cflcontrol="redo", max_redostep_attempts=30,
                      skip_sweep=tuple(d != axis for d in range(3)))
    ob = oracle_lib.OracleBlock(setup, rough_state(setup, seed, mach), None, None)
    ob.fill_guards()
    sim = Simulation(setup)
    sim.upload(ob.u)
    sim.update_boundaries()
    for k in range(6):                     # a redone step counts as one of them
        ob.run(1)
        sim.run(1)
        st = sim.time_state
        assert (st.t, st.dt, st.nstep, st.redone) == (ob.state.t, ob.state.dt, ob.state.nstep, ob.state.redone), k
    gu, _, _ = sim.download()
    assert_bitexact(gu, ob.u, f"{lim} {seed}")
    sim.close()


@pytest.mark.parametrize("n,nb", [((248, 5, 4), 4), ((249, 5, 4), 4), ((5, 248, 4), 4), ((250, 6, 6), 3), ((251, 5, 4), 3),
                                  ((12, 7, 6), 6), ((3, 9, 4), 4), ((2, 8, 2), 2)])
def test_lengths_at_the_lines_of_the_rule(gpu_lib, oracle_lib, n, nb):
    """The longest pencil that the CTA holds with its guard cells and one cell
    more, other guard widths, and pencils shorter than the guard width (both of
    the latter two go stage by stage)."""
    setup = setup_for("hd", n=n, lim="moncen", bnd=(R, O, RO), nb=nb)
    ob = oracle_lib.OracleBlock(setup, random_state(setup, seed=6)[0], None, None)
    ob.fill_guards()
    sim = Simulation(setup)
    sim.upload(ob.u)
    sim.update_boundaries()
    for k in range(3):
        sim.run(1)
        ob.run(1)
        gu, _, _ = sim.download()
        core = tuple(slice(g, g + m) for g, m in zip(setup.guards[::-1], setup.n[::-1]))
        assert_bitexact(np.ascontiguousarray(gu[core]), np.ascontiguousarray(ob.u[core]), f"{n} step {k}")
    sim.close()


@pytest.mark.parametrize("phys,bnd", [("hd", (OR, R, O)), ("hd", (P, P, P)), ("mhd", (P, P, P))])
def test_graphs_of_either_parity(gpu_lib, phys, bnd):
    """A captured step reads one of the two state buffers.  Single sweeps and the
    step that follows an upload (launched one by one for an open block) leave the
    state in the other: steps replayed in any order of the two must equal steps
    launched one by one."""
    setup = setup_for(phys, n=(24, 18, 14), lim="moncen", bnd=bnd)
    state = random_state(setup, seed=7)
    sims = [Simulation(setup), Simulation(setup)]
    sims[1].use_graph()
    start = sims[0].time_state
    for sim in sims:
        for what in ("upload", "run", "run", "sweep", "run", "upload", "run", "run", "sweep", "sweep", "run", "upload", "run",
                     "run"):
            if what == "upload":
                sim.upload(*state)
                sim.time_state = start
            elif what == "sweep":
                sim.sweep(2, 1e-3, 1.0)
            else:
                sim.run(2)
    (u, b, psi), (gu, gb, gp) = (sim.download() for sim in sims)
    assert_bitexact(gu, u, "u")
    if setup.magnetic:
        assert_bitexact(gb, b, "b")
        assert_bitexact(gp, psi, "psi")
    for sim in sims:
        sim.close()
