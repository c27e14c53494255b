"""The persistent GMRES cycle at the sizes where its layout changes: fewer
nodes than a CTA's eight, a ragged last CTA, one block group to several per
node, the basis in and out of shared memory, restarts of one column and of the
largest size. The true residual, formed here from the matrix in goal's CSR
order, is checked against the requested tolerance, and a second solve against
the first bit for bit."""
import numpy as np
import pytest

from oracle import oracle as O
from goal_gb300 import api
from goal_gb300.mesh import kuhn_cube

pytestmark = pytest.mark.gpu


def _system(n, seed=0):
    mesh = kuhn_cube(n, jitter=0.2, seed=seed)
    d = api.Disc(mesh)
    m = api.Mechanics(d, api.J2, [[200e3, 0.3, 1000.0, 250.0, 1.0]])
    rng = np.random.default_rng(seed)
    U = np.zeros((mesh.num_nodes, 4))
    U[:, 0] = 0.002 * mesh.coords[:, 0]
    U[:, :3] += 1e-4 / n * rng.standard_normal((mesh.num_nodes, 3))
    U[:, 3] = rng.standard_normal(mesh.num_nodes)
    m.set_solution(U)
    s = api.SolInfo(d)
    api.assemble(m, s, api.PRIMAL, jacobian=True, save_states=True)
    bcs = api.Bcs(d, [(0, "xmin", "0.0"), (1, "xmin", "0.0"), (2, "xmin", "0.0"), (0, "xmax", "0.002*t")], [])
    api.set_jac_dbcs(m, s, bcs, 1.0)
    return d, m, s, O.csr_matrix(d.graph(), s.dRdu_csr(), d.num_dofs), -s.R


@pytest.mark.parametrize("precision", [api.FP64, api.MIXED, api.MIXED_F32, api.NESTED_F64])
@pytest.mark.parametrize("n,krylov,inner", [(1, 100, 60), (2, 7, 5), (3, 255, 255), (5, 40, 33), (9, 100, 60),
                                            (14, 60, 20)])
def test_reaches_the_residual(n, krylov, inner, precision):
    d, m, s, A, b = _system(n)
    x, st = api.solve(s, b, params=api.solve_params(krylov_size=krylov, max_iters=20000, tolerance=1e-10,
                                                    precision=precision, inner_iters=inner))
    assert st["converged"]
    assert np.linalg.norm(b - A @ x) <= 1.05e-10 * np.linalg.norm(b)
    again, st2 = api.solve(s, b, params=api.solve_params(krylov_size=krylov, max_iters=20000, tolerance=1e-10,
                                                         precision=precision, inner_iters=inner))
    assert np.array_equal(x, again) and st["iters"] == st2["iters"]


@pytest.mark.parametrize("precision", [api.FP64, api.MIXED, api.NESTED_F64])
def test_two_sweeps_and_one_column(precision):
    """The learned second sweep, and a cycle of one column."""
    d, m, s, A, b = _system(6, seed=2)
    net = api.Learned(seed=1)
    net.train([s], epochs=20, lr=3e-3, num_probes=4, seed=5)
    net.attach(s)
    x, st = api.solve(s, b, params=api.solve_params(krylov_size=50, max_iters=20000, tolerance=1e-10,
                                                    precision=precision, inner_iters=20, precond=api.PRECOND_LEARNED))
    assert st["converged"]
    assert np.linalg.norm(b - A @ x) <= 1.05e-10 * np.linalg.norm(b)
    _, st = api.solve(s, b, params=api.solve_params(krylov_size=1, max_iters=3, tolerance=1e-10, precision=precision,
                                                    inner_iters=1))
    assert st["iters"] == 3 and not st["converged"] and 0.0 < st["rel_res"] < 1.0


def test_iteration_cap_and_zero_right_hand_side():
    d, m, s, A, b = _system(5)
    _, st = api.solve(s, b, params=api.solve_params(krylov_size=100, max_iters=17, tolerance=1e-14))
    assert st["iters"] == 17 and not st["converged"]
    x, st = api.solve(s, np.zeros_like(b), params=api.solve_params(tolerance=1e-10))
    assert st["converged"] and st["iters"] == 0 and not x.any()


@pytest.mark.parametrize("precision,inner", [(api.MIXED, 60), (api.MIXED_F32, 23)])
def test_basis_outside_shared_memory(precision, inner):
    """Enough rows on a CTA that the basis and the matrix stay in device
    memory, with column counts on both sides of a batch."""
    d, m, s, A, b = _system(34, seed=3)
    x, st = api.solve(s, b, params=api.solve_params(krylov_size=60, max_iters=20000, tolerance=1e-9,
                                                    precision=precision, inner_iters=inner))
    assert st["converged"]
    assert np.linalg.norm(b - A @ x) <= 1.05e-9 * np.linalg.norm(b)
