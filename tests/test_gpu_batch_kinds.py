"""Batches that hold blocks extruded along k and general ones (a stage and a CFL launch for each
kind): every case advances as it does alone, time steps included, so the next step of a served
case does not depend on its neighbours.  The number of launches tells which kernels ran.
"""
import pytest
import torch

from wmles_jax_b200 import ConstantMassFlux, KEP, Solver, lowering
from wmles_jax_b200.serving import Batch
from wmles_jax_b200.workloads import channel_gas, channel_mesh, loglaw_prim

pytestmark = pytest.mark.gpu

_metrics = lowering._block_metrics


def general(blk, geom):
    """The block's metrics with one component no zero: the same numbers by the general kernels."""
    M = _metrics(blk, geom)
    M[2, 3, 3, 3] = 1e-300
    return M


def stretched_mesh(n):
    """A channel whose span is not uniform (areas times a factor per k on the extruded path)."""
    import numpy as np
    mesh = channel_mesh(n)
    b = mesh.blocks[0]
    span = np.pi
    b.x_int[2] += 0.3 * (span / n[2]) * np.sin(2.0 * np.pi * b.x_int[2] / span)
    mesh.finalize()
    return mesh


def members(precision, monkeypatch, kinds, mesh_of=channel_mesh):
    gas, out = channel_gas(), []
    for n, kind in kinds:
        monkeypatch.setattr(lowering, "_block_metrics", _metrics if kind == "extruded" else general)
        mesh = mesh_of(n)
        s = Solver(mesh, gas, scheme=KEP(4), sgs="wale", cfl=0.5, constraints=[ConstantMassFlux(0, 1.0)],
                   precision=precision)
        out.append((s, s.init_state(loglaw_prim(gas, mesh, seed=n[0]))))
    monkeypatch.setattr(lowering, "_block_metrics", _metrics)
    return out


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("mesh_of", [channel_mesh, stretched_mesh])
def test_batch_of_both_kinds_is_the_cases_alone(precision, mesh_of, monkeypatch):
    kinds = [((16, 12, 20), "extruded"), ((20, 14, 18), "general"), ((24, 12, 34), "extruded"), ((17, 9, 11), "general")]
    cases = members(precision, monkeypatch, kinds, mesh_of)
    qa = [tuple(q.clone() for q in Q) for _, Q in cases]
    qb = [tuple(torch.empty_like(q) for q in Q) for Q in qa]
    da = [s.max_dt(Q) for (s, _), Q in zip(cases, qa)]
    db = [torch.empty_like(d) for d in da]
    batch = Batch([s for s, _ in cases])
    # per stage one surface launch and one stage launch of each kind, per step one CFL launch of each kind
    assert batch.launches_per_step == 3 * (1 + 2) + 2
    alone = [Q for _, Q in cases]
    for _ in range(3):
        batch.step(qa, qb, da, db)                               # the batch's own time steps
        qa, qb, da, db = qb, qa, db, da
        for m, (s, _) in enumerate(cases):
            alone[m], _ = s.step(alone[m])
            assert torch.equal(alone[m][0], qa[m][0])
            assert torch.equal(s.max_dt(alone[m]), da[m])


@pytest.mark.parametrize("kind", ["extruded", "general"])
def test_batch_of_one_kind_has_one_launch_per_kernel(kind, monkeypatch):
    cases = members("fp64", monkeypatch, [((16, 12, 20), kind), ((12, 10, 9), kind)])
    assert Batch([s for s, _ in cases]).launches_per_step == 3 * 2 + 1
