"""The residual alone, node by node: a node whose gradient is far smaller than the
others' has a row that much smaller, and digits of its own. Its terms are some ten
roundings, in the chain with the Jacobian as in the one without: 64 of FP64's of
the row's largest entry."""
import numpy as np
import pytest

from goal_gb300 import api
from goal_gb300.mesh import Mesh, orient_positive

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", [api.NEOHOOKEAN, api.J2])
@pytest.mark.parametrize("far", [0, 1, 2, 3])
@pytest.mark.parametrize("length", [1.0, 1e3, 1e6])
def test_row_of_a_far_node(length, far, model):
    rng = np.random.default_rng(far)
    base = np.array([[0.0, 0.0, 0.0], [1.0, 0.1, 0.0], [0.2, 1.0, 0.1]])
    tip = np.array([0.3, 0.4, 1.0]) * length
    order = [i for i in range(4) if i != far]
    coords = np.empty((4, 3))
    coords[order], coords[far] = base, tip
    tets = orient_positive(coords, np.array([[0, 1, 2, 3]], np.int32))
    mesh = Mesh(coords=coords, tets=tets, elem_set=np.zeros(1, np.int32), elem_set_names=["a"], node_sets={},
                side_sets={})
    d = api.Disc(mesh)
    m = api.Mechanics(d, model, [[200e3, 0.3, 1000.0, 250.0, 1.0]])
    U = rng.standard_normal((4, 4))
    U[:, :3] = coords @ (1e-3 * rng.standard_normal((3, 3))).T
    m.set_solution(U)
    r, j = api.SolInfo(d), api.SolInfo(d)
    api.assemble(m, r, api.PRIMAL, jacobian=False, save_states=False)
    api.assemble(m, j, api.PRIMAL, jacobian=True, save_states=False)
    R, J = r.R.reshape(4, 4), j.R.reshape(4, 4)
    for n in range(4):
        assert np.abs(R[n, :3] - J[n, :3]).max() <= 64 * 2.0 ** -52 * np.abs(J[n, :3]).max()
