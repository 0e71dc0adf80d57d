"""Rounding of the FP64 upwind residual: the shared divisions of the MUSCL-HLLC flux leave it as close to the
method in extended precision as float64 NumPy, which divides for every quotient, is.
"""
import numpy as np
import pytest

from oracle.wmles_oracle import OracleSolver
from wmles_jax_b200 import Block, CharacteristicFarfield, Mesh, MUSCLHLLC, SlipWall, Solver
from wmles_jax_b200.mesh import Geom, compute_geometry
from wmles_jax_b200.workloads import channel_gas

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(np.finfo(np.longdouble).nmant <= 52, reason="needs an extended type")]


def skewed(n):
    x, y, z = np.meshgrid(*(np.linspace(0.0, 1.0, m + 1) for m in n), indexing="ij")
    w = 2.0 * np.pi
    b = Block("box", np.stack([x + 0.03 * np.sin(w * y) * np.sin(w * z), y + 0.02 * np.sin(w * x),
                               z + 0.02 * np.sin(w * x) * np.cos(w * y)]))
    mesh = Mesh([b])
    for a, d in zip("ijk", np.eye(3)):
        mesh.connect(b, a + "min", b, a + "max", shift=tuple(-d))
    return mesh.finalize()


def extruded(n):
    x, y = np.meshgrid(np.linspace(0.0, 2.0, n[0] + 1), np.linspace(0.0, 1.0, n[1] + 1) ** 1.3, indexing="ij")
    y = y + 0.08 * np.sin(np.pi * x) * (1.0 - y)
    z = np.linspace(0.0, 0.7, n[2] + 1)
    shape = x.shape + z.shape
    b = Block("bump", np.stack([np.broadcast_to(x[..., None], shape), np.broadcast_to(y[..., None], shape),
                                np.broadcast_to(z, shape)]))
    mesh = Mesh([b])
    far = np.array([1.0, 1.0, 0.0, 0.0, channel_gas(Ma_b=0.4).R])
    for face, bc in (("imin", CharacteristicFarfield(far)), ("imax", CharacteristicFarfield(far)),
                     ("jmin", SlipWall()), ("jmax", SlipWall())):
        b.set_bc(face, bc)
    mesh.connect(b, "kmin", b, "kmax", shift=(0.0, 0.0, -0.7))
    return mesh.finalize()


@pytest.mark.parametrize("limiter", ["minmod", "albada"])
@pytest.mark.parametrize("grid", [skewed, extruded])
def test_residual_is_as_exact_as_with_divisions(grid, limiter):
    mesh, gas = grid((22, 17, 27)), channel_gas(Ma_b=0.4, Re_b=5000.0)

    def prim(xc):
        e = np.random.default_rng(7).normal(size=(4,) + xc[0].shape)
        p = gas.R * (1.0 + 0.15 * np.tanh(8.0 * np.cos(6.0 * xc[0]) * np.sin(9.0 * xc[1])))
        return np.stack([1.0 + 0.05 * np.sin(3.0 * xc[0]) + 0.01 * e[3], 0.8 + 0.1 * e[0], 0.1 * e[1], 0.2 + 0.1 * e[2], p])
    kw = dict(scheme=MUSCLHLLC(limiter), sgs="wale", cfl=0.5)
    s, ref = Solver(mesh, gas, **kw), OracleSolver(mesh, gas, **kw)
    Q = s.apply_bcs(s.init_state(prim))
    got = mesh.blocks[0].interior(s.rhs(Q)[0].cpu().numpy())
    q = Q[0].cpu().numpy()
    exact = ref.block_rhs(0, q.astype(np.longdouble), Geom(*compute_geometry(mesh.blocks[0].X.astype(np.longdouble))))
    numpy64 = ref.block_rhs(0, q, mesh.geoms[0])
    assert exact.dtype == np.longdouble
    scale = np.sqrt((exact ** 2).reshape(5, -1).mean(axis=1)).reshape(5, 1, 1, 1)

    def rms(a):
        return float(np.sqrt((((a - exact) / scale) ** 2).mean()))
    # both are sums of some hundred roundings a cell over 50 490 values: their ratio is settled to a few percent
    assert rms(got) <= 1.05 * rms(numpy64)
