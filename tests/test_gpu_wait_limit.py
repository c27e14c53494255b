"""Barriers among blocks that run out of their limit: the call returns its error
status, and the next one, at the usual limit, finds nothing left of it. A limit
of one look is too short for all blocks but the last to arrive."""
import contextlib

import numpy as np
import pytest

from goal_gb300 import api, lib
from goal_gb300.mesh import kuhn_cube

pytestmark = pytest.mark.gpu

ERR_SOLVER, ERR_STATE = 7, 3


@contextlib.contextmanager
def one_look():
    api.check(lib().goal_set_wait_limit(1))
    try:
        yield
    finally:
        api.check(lib().goal_set_wait_limit(0))


def _system(n, learned):
    mesh = kuhn_cube(n, jitter=0.2, seed=1)
    rng = np.random.default_rng(2)
    d = api.Disc(mesh)
    m = api.Mechanics(d, api.J2, [[200e3, 0.3, 1000.0, 250.0, 1.0]])
    U = np.zeros((mesh.num_nodes, 4))
    U[:, 0] = 0.002 * mesh.coords[:, 0]
    U[:, :3] += 2e-4 / n * rng.standard_normal((mesh.num_nodes, 3))
    m.set_solution(U)
    s = api.SolInfo(d)
    api.assemble(m, s, api.PRIMAL, jacobian=True, save_states=True)
    bcs = api.Bcs(d, [(0, "xmin", "0.0"), (1, "xmin", "0.0"), (2, "xmin", "0.0"), (0, "xmax", "0.002*t")], [])
    api.set_jac_dbcs(m, s, bcs, 1.0)
    net = None
    if learned:
        net = api.Learned(seed=1)
        net.train([s], epochs=20, lr=3e-3, num_probes=4, seed=5)
        net.attach(s)
    return d, m, s, net, -s.R


@pytest.mark.parametrize("learned", [False, True])
@pytest.mark.parametrize("precision", [api.FP64, api.MIXED, api.MIXED_F32, api.NESTED_F64])
@pytest.mark.parametrize("n", [4, 12])
def test_solve(n, precision, learned):
    d, m, s, net, b = _system(n, learned)
    p = api.solve_params(krylov_size=60, max_iters=400, tolerance=1e-8, precision=precision, inner_iters=30,
                         precond=api.PRECOND_LEARNED if learned else api.PRECOND_BJ)
    x, st = api.solve(s, b, params=p)
    for _ in range(3):
        with one_look(), pytest.raises(api.GoalError) as e:
            api.solve(s, b, params=p)
        assert e.value.code == ERR_SOLVER and "barrier" in str(e.value)
    again, st2 = api.solve(s, b, params=p)
    assert np.array_equal(x, again) and st["iters"] == st2["iters"]


@pytest.mark.parametrize("n", [3, 16])
def test_disc(n):
    mesh = kuhn_cube(n, jitter=0.2, seed=1)
    colors = api.Disc(mesh).colors()
    for _ in range(3):
        with one_look(), pytest.raises(api.GoalError) as e:
            api.Disc(mesh)
        assert e.value.code == ERR_STATE
    assert np.array_equal(api.Disc(mesh).colors(), colors)
