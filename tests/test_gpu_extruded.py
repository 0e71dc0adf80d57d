"""The stage kernel of blocks extruded along k against the general one and the oracle.

A block is taken for extruded when its metrics say so; one metric component set to a value that
is no zero (1e-300, without effect on any sum) sends the same case through the general kernel.
Both evaluate the same formulas; the extruded one takes areas as row value times a factor per k,
within a few units in the last place of the general one's, and leaves out products with zeros.
So the FP64 residuals agree to the round-off of a flux difference: 64 eps times the largest
face flux over the volume, bounded here by 1e-12 of the largest residual near a wall, where
the fluxes are about 100 times the residual.  Float form: the same bits on a uniform span
(the factor is exactly 1); on a stretched one areas differ by a float's last place, and the
residual by as much as of its own rounding (1e-5 of its largest value, the mixed form's error).
The FP64 time step's rate is arranged with fewer roots and divisions there: about eight more
roundings, bounded by 16 eps; the float form's is the general one's.
"""
import numpy as np
import pytest
import torch

from oracle.wmles_oracle import OracleSolver, init_state
from wmles_jax_b200 import (Block, CharacteristicFarfield, EquilibriumWallModel, Hybrid, KEP, Mesh, MUSCLHLLC, SlipWall,
                            Solver, WallModel, lowering)
from wmles_jax_b200.workloads import channel_gas

pytestmark = pytest.mark.gpu


def bump(n, span):
    """A wavy-wall block (x and y curved, extruded along k with the given k coordinates)."""
    x, y = np.meshgrid(np.linspace(0.0, 2.0, n[0] + 1), np.linspace(0.0, 1.0, n[1] + 1) ** 1.3, indexing="ij")
    y = y + 0.08 * np.sin(np.pi * x) * (1.0 - y)
    x = x + 0.05 * np.sin(2.0 * np.pi * y)
    shape = x.shape + (len(span),)
    return np.stack([np.broadcast_to(x[..., None], shape), np.broadcast_to(y[..., None], shape),
                     np.broadcast_to(span, shape)])


def case(n, scheme, stretched):
    gas = channel_gas(Ma_b=0.3, Re_b=5000.0)
    span = np.linspace(0.0, 0.7, n[2] + 1)
    if stretched:
        span = span + 0.02 * np.sin(2.0 * np.pi * span / 0.7)
    b = Block("bump", bump(n, span))
    mesh = Mesh([b])
    far = np.array([1.0, 1.0, 0.0, 0.0, gas.R])
    b.set_bc("imin", CharacteristicFarfield(far))
    b.set_bc("imax", WallModel(EquilibriumWallModel(), T_wall=None, n_match=2))
    b.set_bc("jmin", WallModel(EquilibriumWallModel(), T_wall=1.05, n_match=1))
    b.set_bc("jmax", SlipWall())
    mesh.connect(b, "kmin", b, "kmax", shift=(0.0, 0.0, -0.7))
    mesh.finalize()

    def prim(xc):
        rng = np.random.default_rng(3)
        e = 0.1 * rng.normal(size=(4,) + xc[0].shape)
        one = np.ones_like(xc[0])
        return np.stack([1.0 + 0.05 * np.sin(3 * xc[0]) + 0.1 * e[3], 0.8 + e[0], e[1], 0.2 + e[2],
                         gas.R * (1.0 + 0.05 * np.cos(4 * xc[1]) * one)])
    return mesh, gas, dict(scheme=scheme, sgs="wale", cfl=0.5), prim


# sizes at the edges of tiles: the smallest block, one tile and one column more, a remainder row
@pytest.mark.parametrize("n", [(3, 3, 3), (5, 8, 32), (6, 9, 33), (4, 17, 70), (20, 7, 45)])
@pytest.mark.parametrize("scheme", [KEP(4), Hybrid(KEP(4)), MUSCLHLLC("minmod")])
@pytest.mark.parametrize("stretched", [False, True])
def test_extruded_kernel_matches_the_general_one(n, scheme, stretched, monkeypatch):
    mesh, gas, kw, prim = case(n, scheme, stretched)
    general = lowering._block_metrics

    def off(blk, geom):
        M = general(blk, geom)
        M[2, 3, 3, 3] = 1e-300                                   # z component of one i face
        return M
    ref = OracleSolver(mesh, gas, **kw)
    R0 = ref.rhs(init_state(ref, prim))[0][:, 3:-3, 3:-3, 3:-3]
    for precision in ("fp64", "mixed"):
        out = []
        for f in (general, off):
            monkeypatch.setattr(lowering, "_block_metrics", f)
            s = Solver(mesh, gas, **kw, precision=precision)
            Q = s.init_state(prim)
            R = s.rhs(Q)[0][:, 3:-3, 3:-3, 3:-3].cpu().numpy()
            Qn, dt = s.step(Q)
            out.append((R, Qn[0].cpu().numpy(), float(dt)))
        (a, qa, da), (b, qb, db) = out
        scale = np.abs(R0).reshape(5, -1).max(axis=1).reshape(5, 1, 1, 1)
        if precision == "fp64":
            assert np.max(np.abs(a - R0) / scale) < 1e-11
            assert np.max(np.abs(a - b) / scale) < 1e-12
            assert np.allclose(qa, qb, rtol=0, atol=1e-13 * np.abs(qb).max())
        elif not stretched:
            assert np.array_equal(a, b) and np.array_equal(qa, qb)
        else:
            assert np.max(np.abs(a - b) / scale) < 1e-5
            da = db = 0.0                                        # areas differ by a float's last place
        assert abs(da - db) <= (16 * np.finfo(float).eps * db if precision == "fp64" else 0.0)


def test_batch_of_extruded_and_general_cases_is_the_cases_alone(monkeypatch):
    """Two launches per stage share one constant-mass-flux reduction."""
    from wmles_jax_b200 import ConstantMassFlux
    from wmles_jax_b200.serving import Batch
    from wmles_jax_b200.workloads import channel_mesh, loglaw_prim
    general = lowering._block_metrics

    def off(blk, geom):
        M = general(blk, geom)
        M[2, 3, 3, 3] = 1e-300
        return M
    gas = channel_gas()
    solvers, states = [], []
    for n, f in (((16, 12, 20), general), ((20, 14, 18), off), ((24, 12, 34), general)):
        monkeypatch.setattr(lowering, "_block_metrics", f)
        mesh = channel_mesh(n)
        s = Solver(mesh, gas, scheme=KEP(4), sgs="wale", cfl=0.5, constraints=[ConstantMassFlux(0, 1.0)])
        solvers.append(s)
        states.append(s.init_state(loglaw_prim(gas, mesh, seed=n[0])))
    alone = [s.step(tuple(q.clone() for q in Q))[0][0] for s, Q in zip(solvers, states)]
    out = [tuple(torch.empty_like(q) for q in Q) for Q in states]
    dts = [s.max_dt(Q) for s, Q in zip(solvers, states)]
    Batch(solvers).step(states, out, dts, [torch.empty_like(d) for d in dts])
    for a, b in zip(alone, out):
        assert torch.equal(a, b[0])
