"""The constant-mass-flux sum: the same bits for every cut of the grid into tiles and chunks, so that
a batch may cut its cases' blocks as suits the batch; and as exact as the state it shifts.
"""
import math

import numpy as np
import pytest
import torch

from wmles_jax_b200 import ConstantMassFlux, KEP, Solver, lowering
from wmles_jax_b200.serving import Batch
from wmles_jax_b200.workloads import channel_gas, channel_mesh, loglaw_prim

pytestmark = pytest.mark.gpu

_metrics = lowering._block_metrics


def general(blk, geom):
    M = _metrics(blk, geom)
    M[2, 3, 3, 3] = 1e-300                                       # no zero: the general kernels, the same numbers
    return M


def solver(n, precision="fp64", target=1.0, **kw):
    gas, mesh = channel_gas(), channel_mesh(n)
    s = Solver(mesh, gas, scheme=KEP(4), sgs="wale", cfl=0.5, constraints=[ConstantMassFlux(0, target)],
               precision=precision, **kw)
    return s, s.init_state(loglaw_prim(gas, mesh, seed=n[1]))


def advance(s, Q, steps=3):
    for _ in range(steps):
        Q, dt = s.step(Q)
    return Q[0], dt


# sets of cuts whose stage kernel is one instance (one CTA of 512 or two of 256 columns in the float form)
@pytest.mark.parametrize("precision,tiles", [("fp64", (None, 0, 1, 2)), ("mixed", (None, 3)), ("mixed", (0, 1, 2))])
@pytest.mark.parametrize("kind", ["extruded", "general"])
@pytest.mark.parametrize("target", [1.0, 0.0])
def test_bits_do_not_depend_on_tiles_and_chunks(precision, tiles, kind, target, monkeypatch):
    monkeypatch.setattr(lowering, "_block_metrics", _metrics if kind == "extruded" else general)
    n = (29, 19, 41)
    first = None
    for tile in tiles:
        for chunk in (None, 7):
            q, dt = advance(*solver(n, precision, target, tile=tile, chunk=chunk))
            if first is None:
                first = (q, dt)
            assert torch.equal(q, first[0]) and torch.equal(dt, first[1]), (tile, chunk)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("target", [1.0, 0.0, 3e-5])
def test_mean_flux_is_the_target_to_rounding(precision, target):
    s, Q = solver((40, 24, 36), precision, target)
    q, _ = advance(s, Q, 2)
    blk, vol = s.mesh.blocks[0], s.host_geoms[0].vol
    x = (blk.interior(q.cpu().numpy())[1] * blk.interior(vol)).ravel()
    total = math.fsum(x.tolist()) / math.fsum(blk.interior(vol).ravel().tolist())
    # every momentum is rounded once by the shift and its product with the volume once here, 34560 of each
    # (their sum stays below one unit of the largest), the shift, the volume's sum and the quotient a few more
    assert abs(total - target) <= 8 * np.finfo(float).eps * np.abs(blk.interior(q.cpu().numpy())[1]).max()


@pytest.mark.parametrize("precision,fixed", [("fp64", 0), ("mixed", 3)])
@pytest.mark.parametrize("kind", ["extruded", "general"])
def test_many_small_cases_are_cut_as_a_batch(precision, fixed, kind, monkeypatch):
    """Sixty cases that would each spread over the GPU alone: the batch cuts them into no more tiles than
    the largest fixed shape does, and each advances as it does alone."""
    monkeypatch.setattr(lowering, "_block_metrics", _metrics if kind == "extruded" else general)
    n, count = (16, 16, 16), 60
    s, Q = solver(n, precision)
    cases = [s] + [solver(n, precision)[0] for _ in range(count - 1)]
    batch = Batch(cases)
    assert batch.ntiles <= Batch([solver(n, precision, tile=fixed)[0] for _ in range(count)]).ntiles
    assert batch.ntiles < count * Batch([s]).ntiles
    qa = [tuple(q.clone() for q in Q) for _ in cases]
    qb = [tuple(torch.empty_like(q) for q in Q) for _ in cases]
    da = [s.max_dt(Q) for _ in cases]
    db = [torch.empty_like(d) for d in da]
    for _ in range(2):
        batch.step(qa, qb, da, db)
        qa, qb, da, db = qb, qa, db, da
    q, _ = advance(s, Q, 2)
    dt = s.max_dt((q,))
    for m in range(count):
        assert torch.equal(qa[m][0], q) and torch.equal(da[m], dt)
