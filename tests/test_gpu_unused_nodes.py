"""Nodes that no element uses, in the middle and at the end of the numbering: each
has a diagonal block of zeros, and the rows of the others are the bits of the mesh
without them."""
import numpy as np
import pytest

from goal_gb300 import api
from goal_gb300.mesh import Mesh, kuhn_cube

pytestmark = pytest.mark.gpu


def _assembled(mesh, U, mode, overwrite, colored):
    d = api.Disc(mesh)
    m = api.Mechanics(d, api.NEOHOOKEAN, [[1000.0, 0.25, 0.0, 0.0, 1.0]])
    m.set_solution(U)
    s = api.SolInfo(d)
    api.assemble(m, s, mode, jacobian=True, save_states=False, overwrite=overwrite, colored=colored)
    return d.graph(), s.R.reshape(-1, 4), s.dRdu_csr()


@pytest.mark.parametrize("mode", [api.PRIMAL, api.ADJOINT])
@pytest.mark.parametrize("overwrite,colored", [(True, False), (False, False), (True, True)])
@pytest.mark.parametrize("unused", [[0], [17], [64], [0, 1, 30, 67, 68]])  # numbers among all nodes
def test_unused_nodes(unused, overwrite, colored, mode):
    g = kuhn_cube(3, jitter=0.2, seed=1)  # 64 nodes
    unused = np.array(unused)
    N = g.num_nodes + len(unused)
    at = np.setdiff1d(np.arange(N), unused)
    coords = np.full((N, 3), 7.0)
    coords[at] = g.coords
    mesh = Mesh(coords=coords, tets=at[g.tets].astype(np.int32), elem_set=g.elem_set, elem_set_names=g.elem_set_names,
                node_sets={}, side_sets={})
    U = np.zeros((N, 4))
    U[at] = 1e-3 * np.random.default_rng(2).standard_normal((g.num_nodes, 4))
    (rp, ci), R, A = _assembled(mesh, U, mode, overwrite, colored)
    (rp0, ci0), R0, A0 = _assembled(g, U[at], mode, overwrite, colored)
    rows = np.repeat(np.arange(4 * N), np.diff(rp)) // 4
    used = np.isin(rows, at)
    assert np.array_equal(at[ci0 // 4] * 4 + ci0 % 4, ci[used]) and np.array_equal(A0, A[used])
    assert np.array_equal(R0, R[at]) and not R[unused].any()
    assert np.array_equal(ci[~used] // 4, rows[~used]) and not A[~used].any() and (~used).sum() == 16 * len(unused)
