"""Which blocks take the extruded kernels, and the parts of those kernels that the comparisons of
test_gpu_extruded.py do not reach: wall-modelled k faces, the small tiles of the float form, a step on a
stretched span in the float form.

A batch of a case and its copy with a metric component that is no zero has two stage launches a stage
exactly when the two are of different kinds, so when the case itself is taken for extruded.
"""
import numpy as np
import pytest

from oracle.wmles_oracle import OracleSolver, init_state
from wmles_jax_b200 import Block, EquilibriumWallModel, Hybrid, KEP, Mesh, MUSCLHLLC, SlipWall, Solver, WallModel, lowering
from wmles_jax_b200.serving import Batch
from wmles_jax_b200.workloads import channel_case, channel_gas, naca_case, ramp_case

pytestmark = pytest.mark.gpu

ONE_KIND, BOTH_KINDS = 3 * 2 + 1, 3 * 3 + 2                      # launches of a step without an inflow
_metrics = lowering._block_metrics


def general(blk, geom):
    M = _metrics(blk, geom)
    M[2, 3, 3, 3] = 1e-300                                       # no zero: the general kernels, the same numbers
    return M


def pair(monkeypatch, mesh, gas, kw, **opts):
    """The case, and the same through the general kernels."""
    out = []
    for f in (_metrics, general):
        monkeypatch.setattr(lowering, "_block_metrics", f)
        out.append(Solver(mesh, gas, **kw, **opts))
    monkeypatch.setattr(lowering, "_block_metrics", _metrics)
    return out


def bump(n, stretched, kwalls=False):
    gas = channel_gas(Ma_b=0.3, Re_b=5000.0)
    x, y = np.meshgrid(np.linspace(0.0, 2.0, n[0] + 1), np.linspace(0.0, 1.0, n[1] + 1) ** 1.3, indexing="ij")
    y = y + 0.08 * np.sin(np.pi * x) * (1.0 - y)
    x = x + 0.05 * np.sin(2.0 * np.pi * y)
    z = np.linspace(0.0, 0.7, n[2] + 1)
    if stretched:
        z = z + 0.02 * np.sin(2.0 * np.pi * z / 0.7)
    shape = x.shape + z.shape
    b = Block("bump", np.stack([np.broadcast_to(x[..., None], shape), np.broadcast_to(y[..., None], shape),
                                np.broadcast_to(z, shape)]))
    mesh = Mesh([b])
    wall = EquilibriumWallModel()
    for face in ("imin", "imax", "jmax"):
        b.set_bc(face, SlipWall())
    b.set_bc("jmin", WallModel(wall, T_wall=1.05, n_match=1))
    if kwalls:
        b.set_bc("kmin", WallModel(wall, T_wall=None, n_match=1))
        b.set_bc("kmax", WallModel(wall, T_wall=0.97, n_match=2))
    else:
        mesh.connect(b, "kmin", b, "kmax", shift=(0.0, 0.0, -0.7))
    mesh.finalize()

    def prim(xc):
        e = 0.1 * np.random.default_rng(5).normal(size=(4,) + xc[0].shape)
        return np.stack([1.0 + 0.05 * np.sin(3.0 * xc[0]) + 0.1 * e[3], 0.8 + e[0], e[1], 0.2 + e[2],
                         gas.R * (1.0 + 0.05 * np.cos(4.0 * xc[1]))])
    return mesh, gas, dict(sgs="wale", cfl=0.5), prim


@pytest.mark.parametrize("stretched", [False, True])
@pytest.mark.parametrize("n", [(3, 3, 3), (5, 8, 32), (6, 9, 33), (4, 17, 70), (20, 7, 45)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_bump_is_taken_for_extruded(n, stretched, precision, monkeypatch):
    mesh, gas, kw, _ = bump(n, stretched)
    a, b = pair(monkeypatch, mesh, gas, dict(kw, scheme=KEP(4)), precision=precision)
    assert Batch([a, b]).launches_per_step == BOTH_KINDS
    assert Batch([a]).launches_per_step == Batch([b]).launches_per_step == ONE_KIND


def test_workloads_are_extruded(monkeypatch):
    for mesh, gas, kw in (channel_case(2, n=(16, 12, 10))[:3], naca_case(scale=4)[:3]):
        a, b = pair(monkeypatch, mesh, gas, kw)
        assert Batch([a]).launches_per_step == ONE_KIND          # all its blocks are of one kind
        assert Batch([a, b]).launches_per_step == BOTH_KINDS     # and not of the general one
    mesh, gas, kw = ramp_case((48, 24, 16))[:3]
    a, b = pair(monkeypatch, mesh, gas, kw)
    assert Batch([a, b]).launches_per_step - 2 * (Batch([a]).launches_per_step - ONE_KIND) == BOTH_KINDS


@pytest.mark.parametrize("stretched", [False, True])
@pytest.mark.parametrize("scheme", [KEP(4), Hybrid(KEP(4)), MUSCLHLLC("minmod")])
def test_wall_modelled_k_faces(scheme, stretched, monkeypatch):
    mesh, gas, kw, prim = bump((9, 10, 35), stretched, kwalls=True)
    kw = dict(kw, scheme=scheme)
    ref = OracleSolver(mesh, gas, **kw)
    R0 = mesh.blocks[0].interior(ref.rhs(init_state(ref, prim))[0])
    scale = np.abs(R0).reshape(5, -1).max(axis=1).reshape(5, 1, 1, 1)
    for precision, to_oracle in (("fp64", 1e-11), ("mixed", 1e-4)):
        a, b = pair(monkeypatch, mesh, gas, kw, precision=precision)
        assert Batch([a, b]).launches_per_step == BOTH_KINDS
        ra, rb = (mesh.blocks[0].interior(s.rhs(s.init_state(prim))[0].cpu().numpy()) for s in (a, b))
        # as in test_gpu_extruded.py: the parity bound, 64 eps of the largest face flux, a float's last place
        assert np.max(np.abs(ra - R0) / scale) < to_oracle
        assert np.max(np.abs(ra - rb) / scale) <= (1e-12 if precision == "fp64" else 1e-5 if stretched else 0.0)


@pytest.mark.parametrize("tile", [0, 1, 2, 3])
@pytest.mark.parametrize("scheme", [KEP(4), Hybrid(KEP(4)), MUSCLHLLC("albada")])
def test_fixed_tiles_of_the_float_form(tile, scheme, monkeypatch):
    mesh, gas, kw, prim = bump((7, 21, 43), False)
    a, b = pair(monkeypatch, mesh, gas, dict(kw, scheme=scheme), precision="mixed", tile=tile)
    (qa, da), (qb, db) = (s.step(s.init_state(prim)) for s in (a, b))
    assert np.array_equal(qa[0].cpu().numpy(), qb[0].cpu().numpy()) and float(da) == float(db)


@pytest.mark.parametrize("scheme", [KEP(4), Hybrid(KEP(4)), MUSCLHLLC("minmod")])
def test_step_on_a_stretched_span_in_the_float_form(scheme, monkeypatch):
    mesh, gas, kw, prim = bump((11, 17, 37), True)
    kw = dict(kw, scheme=scheme)
    a, b = pair(monkeypatch, mesh, gas, kw, precision="mixed")
    ref = OracleSolver(mesh, gas, **kw)
    R0 = mesh.blocks[0].interior(ref.rhs(init_state(ref, prim))[0])
    (qa, da), (qb, db) = (s.step(s.init_state(prim)) for s in (a, b))
    # the rate holds some twenty float roundings of areas either way
    assert abs(float(da) - float(db)) <= 32 * np.finfo(np.float32).eps * float(db)
    # a step moves the state by dt times a mean of three residuals, each within 1e-5 of its largest value
    # (test_gpu_extruded.py) of the other kernel's; the residuals of the later stages stay below twice the first's
    bound = float(db) * (2 * 1e-5 + 32 * np.finfo(np.float32).eps) * 2 * np.abs(R0).reshape(5, -1).max(axis=1)
    d = np.abs(mesh.blocks[0].interior((qa[0] - qb[0]).cpu().numpy())).reshape(5, -1).max(axis=1)
    assert (d <= bound).all()
