"""Side sets of the discretization build: the nodes that a traction reaches are
those of its set, whatever the order of its sides."""
import numpy as np
import pytest

from goal_gb300 import api
from goal_gb300.mesh import Mesh, kuhn_cube

pytestmark = pytest.mark.gpu


def _with(mesh, **sets):
    return Mesh(coords=mesh.coords, tets=mesh.tets, elem_set=mesh.elem_set, elem_set_names=mesh.elem_set_names,
                node_sets=mesh.node_sets, side_sets={**mesh.side_sets, **sets})


def _loaded(mesh, name):
    d = api.Disc(mesh)
    m = api.Mechanics(d, api.NEOHOOKEAN, [[1000.0, 0.25, 0.0, 0.0, 1.0]])
    s = api.SolInfo(d)
    api.assemble(m, s, api.PRIMAL, jacobian=False, save_states=False)
    before = s.R.copy()
    api.set_tbcs(m, s, api.Bcs(d, [], [(name, "0.0", "0.0", "1.0")]), 1.0)
    return s.R - before


@pytest.mark.parametrize("n", [1, 2, 14])  # one, two and three digits of the sort's
def test_traction_reaches_the_set_and_no_more(n):
    mesh = kuhn_cube(n)
    tris = mesh.side_sets["zmax"]
    shuffled = tris[np.random.default_rng(n).permutation(len(tris))]
    R = _loaded(_with(mesh, mixed=shuffled, none=np.zeros((0, 3), np.int32)), "mixed").reshape(-1, 4)
    on = np.zeros(mesh.num_nodes, bool)
    on[tris.ravel()] = True
    assert np.all(R[~on] == 0.0) and np.all(R[on, 2] != 0.0)
    assert abs(abs(R[:, 2].sum()) - 1.0) < 1e-12  # a unit traction on a unit face
    assert np.allclose(R, _loaded(mesh, "zmax").reshape(-1, 4), rtol=0, atol=1e-15)


def test_time_of_many_small_sets_is_their_own():
    """Two sides in each of 500 sets, on a mesh of 2,200 nodes and one of 118,000:
    the same work. (7 and 8 ms; 10 and more times as long on the larger mesh if
    each set went over its nodes.)"""
    def best(n):
        mesh = kuhn_cube(n)
        tris = mesh.side_sets["zmax"]
        mesh = Mesh(coords=mesh.coords, tets=mesh.tets, elem_set=mesh.elem_set, elem_set_names=mesh.elem_set_names,
                    node_sets={}, side_sets={f"s{i}": tris[i % 200:i % 200 + 2] for i in range(500)})
        return min(api.Disc(mesh).build_times()["sets"] for _ in range(4))

    assert best(48) < 4.0 * best(12)
