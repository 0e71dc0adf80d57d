"""The wall model's Newton iteration on the device over its constants: the friction velocity is the
reference's iterate (wmles/wall_model.py:19-40) for any kappa, B and number of iterations, settled or not, on
both sides of the Reynolds numbers at which the start changes.
"""
import numpy as np
import pytest

from oracle.wmles_oracle import OracleSolver
from wmles_jax_b200 import Block, EquilibriumWallModel, Gas, KEP, Mesh, SlipWall, Solver, WallModel
from wmles_jax_b200 import _native as N

pytestmark = pytest.mark.gpu

# (kappa, B, iterations): the usual constants with the usual number, the last one that keeps the reference's
# start, few and many; the edges of the range that takes the other start; and constants for which the
# reference does not settle in thirty iterations
RANGE = [(0.41, 5.2, 30), (0.41, 5.2, 29), (0.41, 5.2, 100), (0.41, 5.2, 6), (0.41, 5.2, 1), (0.41, 5.2, 0),
         (0.384, 4.17, 30), (0.41, -3.0, 30), (0.6, 5.2, 30), (0.6, 20.0, 30), (0.601, 20.0, 30), (0.3, -15.0, 30),
         (0.3, -16.0, 30), (0.8, 29.0, 30), (1.0, -5.0, 30), (1.5, 5.2, 30), (2.0, 3.3, 30), (4.0, 12.0, 31), (0.05, 5.2, 30)]
UNSETTLED = {(0.41, 5.2, 6), (0.41, 5.2, 1), (0.8, 29.0, 30), (2.0, 3.3, 30), (4.0, 12.0, 31)}


@pytest.mark.parametrize("kappa,B,n_iter", RANGE)
def test_friction_is_the_reference_iterate(kappa, B, n_iter):
    gas = Gas(R=1e10, mu_ref=1e-9, T_ref=1.0, S_suth=0.4)        # pressure far above the stagnation pressures here
    n, h = (16, 4, 24), 0.05
    axes = [np.arange(n[0] + 1) * 0.1, np.arange(n[1] + 1) * 2.0 * h, np.arange(n[2] + 1) * 0.1]
    b = Block("wall", np.stack(np.meshgrid(*axes, indexing="ij")))
    mesh = Mesh([b])
    mesh.connect(b, "imin", b, "imax", shift=(-0.1 * n[0], 0.0, 0.0))
    mesh.connect(b, "kmin", b, "kmax", shift=(0.0, 0.0, -0.1 * n[2]))
    b.set_bc("jmin", WallModel(EquilibriumWallModel(kappa, B, n_iter), T_wall=1.0, n_match=1))
    b.set_bc("jmax", SlipWall())
    mesh.finalize()
    # Re_h = h U rho / mu = 5e7 U, one value per face
    Reh = 10.0 ** np.linspace(0.0, 13.0, n[0] * n[2]).reshape(n[0], n[2])
    Reh.ravel()[:6] = [624.999999, 625.0, 625.000001, 9.99999e11, 1e12, 1.00001e12]
    U = np.pad(Reh / 5e7, 3, mode="wrap")[:, None, :]

    def prim(xc):
        one = np.ones_like(xc[0])
        return np.stack([one, U * one, 0.0 * one, 0.0 * one, 1e10 * one])
    kw = dict(scheme=KEP(2), sgs=None, cfl=0.5)
    s, ref = Solver(mesh, gas, **kw), OracleSolver(mesh, gas, **kw)
    Q = s.init_state(prim)
    s.status(clear=True)
    tau, _ = s.wall_stats(Q)[("wall", "jmin")]
    want, _ = ref.wall_stats(tuple(q.cpu().numpy() for q in Q))[("wall", "jmin")]
    # tau = rho (U / u+)^2: twice the error of u+, which is some 64 eps where the iteration settles (the rounding
    # of F's terms over u+ dF), and where it does not, that of each step carried on by a contraction
    np.testing.assert_allclose(tau, want, rtol=1e-12)
    assert bool(s.status() & N.ST_WALL) == ((kappa, B, n_iter) in UNSETTLED)
