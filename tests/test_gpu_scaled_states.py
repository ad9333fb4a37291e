"""States whose operands leave the range in which the kernels' branch-free
quotients (pk_quotient.cuh) are proven: the threads that hold them redo their
cells in IEEE operations, and the result must be the oracle's, bit for bit.

Units scaled far down and far up, and fields that fade through the whole
exponent range (values from 1e-100 to 1e-300 between ordinary ones, so that
some threads of a warp redo their cells and others do not)."""
import numpy as np
import pytest

from helpers import assert_bitexact, random_state, setup_for
from piernik_b200.sim import Simulation

pytestmark = pytest.mark.gpu


def scaled(setup, how, seed=3):
    u, b, psi = random_state(setup, seed=seed)
    if how == "fading":
        rng = np.random.default_rng(seed)
        for f, (kind, gam) in enumerate(setup.fluids):
            o = sum(4 if k == "dst" else 5 for k, _ in setup.fluids[:f])
            tiny = 10.0 ** rng.uniform(-300, -100, u.shape[:3] + (3,)) * rng.choice([-1.0, 0.0, 1.0], u.shape[:3] + (3,))
            u[..., o + 1:o + 4] = np.where(rng.random(u.shape[:3] + (1,)) < 0.7, tiny, u[..., o + 1:o + 4])
        if setup.magnetic:
            small = 10.0 ** rng.uniform(-300, -100, b.shape) * rng.choice([-1.0, 0.0, 1.0], b.shape)
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
