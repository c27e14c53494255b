"""The solver where its persistent cycle does not hold everything: systems beyond
its limits, which run a kernel per step (all precisions, one and two sweeps), and
FP64 systems whose basis stays in device memory. The true residual is formed here
from the matrix in goal's CSR order."""
import functools

import numpy as np
import pytest

from oracle import oracle as O
from goal_gb300 import api, lib
from goal_gb300.mesh import kuhn_cube

pytestmark = pytest.mark.gpu


@functools.lru_cache(maxsize=1)
def _system(n):
    mesh = kuhn_cube(n, jitter=0.2, seed=3)
    d = api.Disc(mesh)
    m = api.Mechanics(d, api.J2, [[200e3, 0.3, 1000.0, 250.0, 1.0]])
    rng = np.random.default_rng(3)
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


@functools.lru_cache(maxsize=1)
def _net():
    d, m, s, _, _ = _system.__wrapped__(6)
    net = api.Learned(seed=1)
    net.train([s], epochs=40, lr=3e-3, num_probes=8, seed=5)
    return net


def _solve(n, learned, **params):
    d, m, s, A, b = _system(n)
    if learned:
        _net().attach(s)
    p = api.solve_params(precond=api.PRECOND_LEARNED if learned else api.PRECOND_BJ, **params)
    before = lib().goal_launch_count()
    x, st = api.solve(s, b, params=p)
    launches = lib().goal_launch_count() - before
    true = float(np.linalg.norm(b - A @ x) / np.linalg.norm(b))
    assert abs(true - st["rel_res"]) <= 1e-6 * true + 1e-14
    return st, launches


# 185,193 nodes: above the limits of FP64 arithmetic and of two sweeps; 373,248: above all
@pytest.mark.parametrize("n,precision,learned",
                         [(56, api.FP64, False), (56, api.FP64, True), (56, api.NESTED_F64, False),
                          (56, api.NESTED_F64, True), (56, api.MIXED, True), (56, api.MIXED_F32, True),
                          (71, api.MIXED, False), (71, api.MIXED_F32, False)])
def test_kernel_per_step(n, precision, learned):
    if precision == api.FP64:  # thousands of iterations to the end: two restarts and a half
        st, launches = _solve(n, learned, krylov_size=60, max_iters=150, tolerance=1e-10, precision=precision)
        assert st["iters"] == 150 and st["rel_res"] < 0.9
        assert launches >= 3 * st["iters"]
        return
    st, launches = _solve(n, learned, krylov_size=100, max_iters=400, tolerance=1e-8, precision=precision,
                          inner_iters=60)
    assert st["converged"]
    assert launches >= 3 * st["inner_iters"]


@pytest.mark.parametrize("learned", [False, True])
@pytest.mark.parametrize("precision,krylov,inner", [(api.FP64, 100, 1), (api.FP64, 255, 1), (api.NESTED_F64, 100, 60),
                                                    (api.NESTED_F64, 40, 255)])
def test_fp64_basis_outside_shared_memory(precision, krylov, inner, learned):
    st, launches = _solve(22, learned, krylov_size=krylov, max_iters=20000, tolerance=1e-9, precision=precision,
                          inner_iters=inner)
    assert st["converged"]
    assert launches < 40 * max(1, st["iters"] if precision == api.NESTED_F64 else st["iters"] // krylov + 1)
