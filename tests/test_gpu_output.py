"""Derived fields and plane statistics at the edges of their kernels' tiles and chunks (blocks
narrower and wider than a tile, one column over, chunks shorter than a CTA), on extruded and skewed
blocks, against the oracle.  Tolerances: those of the golden comparisons (1e-11 of a field's
largest value: FP64 gradients, ratios and differences of them; 1e-12 for means of some
thousand values)."""
import numpy as np
import pytest
import torch

from oracle.wmles_oracle import OracleSolver, derived_fields as oracle_derived, plane_means
from test_gpu_extruded import case
from wmles_jax_b200 import KEP, Block, Mesh, SlipWall, Solver
from wmles_jax_b200.output import derived_fields
from wmles_jax_b200.stats import KEYS, PlaneStats

pytestmark = pytest.mark.gpu

SIZES = [(4, 5, 4), (5, 33, 4), (37, 4, 33), (6, 9, 65), (70, 6, 16)]


def skewed(n):
    """A slip-walled box whose faces vary along k (the general path)."""
    mesh, gas, kw, prim = case(n, KEP(4), False)
    X = np.array(mesh.blocks[0].x_int)
    X[0] += 0.03 * X[2] * X[1]
    b = Block("skewed", X)
    for face in ("imin", "imax", "jmin", "jmax", "kmin", "kmax"):
        b.set_bc(face, SlipWall())
    m = Mesh([b])
    m.finalize()
    return m, gas, kw, prim


@pytest.mark.parametrize("general", (False, True))
@pytest.mark.parametrize("n", SIZES)
def test_derived_and_plane_means(n, general):
    mesh, gas, kw, prim = skewed(n) if general else case(n, KEP(4), False)
    s, o = Solver(mesh, gas, **kw), OracleSolver(mesh, gas, **kw)
    Q = s.init_state(prim)
    Qh = tuple(q.cpu().numpy() for q in Q)
    want, got = oracle_derived(o, Qh)[0], derived_fields(s, Q)[0]
    for k, v in got.items():
        assert np.abs(v - want[k]).max() <= 1e-11 * np.abs(want[k]).max(), k
    ps = PlaneStats(mesh, s)
    ps.accumulate(Q)
    _, avg = ps.result()
    ref = plane_means(gas, mesh.blocks[0], Qh[0])
    for a, b in (("u", "u"), ("v", "v"), ("w", "w"), ("u", "v"), ("u", "w"), ("v", "w")):
        ref[a + b] = ref[a + b] - ref[a] * ref[b]
    for k in KEYS:
        np.testing.assert_allclose(avg[k], ref[k], rtol=1e-12, atol=1e-13, err_msg=k)
