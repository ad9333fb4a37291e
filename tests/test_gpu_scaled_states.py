"""States whose operands leave the range in which the kernels' branch-free
quotients (pk_quotient.cuh) are proven: the threads that hold them redo their
cells in IEEE operations, and the result must be the oracle's, bit for bit.

Units scaled far down and far up, and fields that fade through the whole
exponent range (values from 1e-100 to 1e-322 between ordinary ones, so that
some threads of a warp redo their cells and others do not)."""
import numpy as np
import pytest

from helpers import assert_bitexact, random_state, setup_for
from piernik_b200.config import BND_OUT, BND_REF
from piernik_b200.sim import Simulation

pytestmark = pytest.mark.gpu


def scaled(setup, how, seed=3):
    u, b, psi = random_state(setup, seed=seed)
    if setup.fluids[-1][0] == "dst":       # moving one way: diverging dust meets the reference's 0 / 0
        u[..., -3:] = u[..., -4:-3] * (0.3 + 0.1 * np.abs(u[..., -3:]))
    if how == "fading":
        rng = np.random.default_rng(seed)
        for f, (kind, gam) in enumerate(setup.fluids):
            if kind == "dst":
                continue
            o = sum(4 if k == "dst" else 5 for k, _ in setup.fluids[:f])
            tiny = 10.0 ** rng.uniform(-322, -100, u.shape[:3] + (3,)) * rng.choice([-1.0, 0.0, 1.0], u.shape[:3] + (3,))
            u[..., o + 1:o + 4] = np.where(rng.random(u.shape[:3] + (1,)) < 0.7, tiny, u[..., o + 1:o + 4])
        if setup.magnetic:
            small = 10.0 ** rng.uniform(-322, -100, b.shape) * rng.choice([-1.0, 0.0, 1.0], b.shape)
            b[...] = np.where(rng.random(b.shape) < 0.6, small, b)
        return u, b, psi
    r = {"down": 2.0**-460, "up": 2.0**460}[how]      # densities, momenta, energies; fields by the root
    u *= r
    if setup.magnetic:
        b *= np.sqrt(r)
        psi *= np.sqrt(r)
    return u, b, psi


def _check(oracle_lib, setup, how):
    setup = setup.replace(use_smalld=False, use_smallei=False)
    ob = oracle_lib.OracleBlock(setup, *scaled(setup, how))
    ob.fill_guards()
    sim = Simulation(setup)
    sim.upload(ob.u, ob.b, ob.psi)
    sim.update_boundaries()
    for axis in (0, 1, 2, 0):
        if setup.n[axis] == 1:
            continue
        dt, c = ob.timestep_raw()
        assert sim.timestep_raw() == (dt, c) and np.isfinite(dt) and dt > 0
        ob.sweep(axis, 0.5 * dt, 1.0)
        sim.sweep(axis + 1, 0.5 * dt, 1.0)
        gu, gb, gp = sim.download()
        assert np.isfinite(ob.u).all()
        assert_bitexact(gu, ob.u, f"u {how} axis {axis}")
        if setup.magnetic:
            assert_bitexact(gb, ob.b, f"b {how} axis {axis}")
            assert_bitexact(gp, ob.psi, f"psi {how} axis {axis}")
    sim.close()


@pytest.mark.parametrize("how", ["down", "up", "fading"])
@pytest.mark.parametrize("phys", ["hd", "mhd"])
def test_weno3(gpu_lib, oracle_lib, phys, how):
    _check(oracle_lib, setup_for(phys, n=(33, 18, 12), lim="weno3", w_epsilon=1e-10), how)


@pytest.mark.parametrize("how", ["down", "up", "fading"])
@pytest.mark.parametrize("phys,lim", [("hd", "vanleer"), ("hd", "moncen"), ("mhd", "vanleer"), ("mhd", "superbee")])
def test_linear(gpu_lib, oracle_lib, phys, lim, how):
    """utoq, the slopes, both solvers, the floors and the CFL reduction: the tile
    of small blocks."""
    _check(oracle_lib, setup_for(phys, n=(33, 18, 12), lim=lim), how)


@pytest.mark.parametrize("how", ["down", "up", "fading"])
@pytest.mark.parametrize("phys,n,kw", [("hd", (64, 64, 48), {}), ("mhd", (64, 64, 48), {}),     # staged whole pencils
                                       ("hd", (300, 130, 1), {}), ("mhd", (300, 130, 1), {}),   # chunks
                                       ("hd", (40, 20, 16), {"bnd": ((BND_OUT, BND_REF),) * 3})])   # an open box
def test_other_kernels(gpu_lib, oracle_lib, phys, n, kw, how):
    _check(oracle_lib, setup_for(phys, n=n, lim="vanleer", **kw), how)


@pytest.mark.parametrize("how", ["down", "up", "fading"])
def test_three_fluids(gpu_lib, oracle_lib, how):
    """More components than cross the barriers in registers, dust among them."""
    setup = setup_for("mhd", n=(20, 12, 8), lim="vanleer")
    setup = setup.replace(fluids=[("ion", 5.0 / 3.0), ("neu", 1.4), ("dst", -1.0)])
    _check(oracle_lib, setup, how)


@pytest.mark.parametrize("how", ["down", "up", "fading"])
@pytest.mark.parametrize("phys", ["hd", "mhd"])
def test_unsplit(gpu_lib, oracle_lib, phys, how):
    setup = setup_for(phys, n=(33, 18, 12), lim="vanleer", solver="unsplit", cfl=0.3, cfl_glm=0.3, use_smalld=False,
                      use_smallei=False)
    ob = oracle_lib.OracleBlock(setup, *scaled(setup, how))
    ob.fill_guards()
    sim = Simulation(setup)
    sim.upload(ob.u, ob.b, ob.psi)
    assert ob.run(2) == 0
    sim.run(2)
    gu, gb, _ = sim.download()
    assert np.isfinite(ob.u).all()
    assert_bitexact(gu, ob.u, f"u {how}")
    if setup.magnetic:
        assert_bitexact(gb, ob.b, f"b {how}")
    sim.close()
