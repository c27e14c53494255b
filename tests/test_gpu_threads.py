"""Several threads at once: the results of one thread, bit for bit."""
import threading

import numpy as np
import pytest

from goal_gb300 import api
from goal_gb300.mesh import kuhn_cube

pytestmark = pytest.mark.gpu

ROW = [200e3, 0.3, 1000.0, 250.0, 1.0]


def _together(jobs):
    """Runs the functions in a thread each, from a common start; their results."""
    out, start = [None] * len(jobs), threading.Barrier(len(jobs))

    def work(i):
        start.wait()
        try:
            out[i] = jobs[i]()
        except Exception as e:  # noqa: BLE001 (handed to the test below)
            out[i] = e

    ts = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for r in out:
        if isinstance(r, Exception):
            raise r
    return out


def _state(mesh, seed):
    rng = np.random.default_rng(seed)
    U = 1e-3 / 6 * rng.standard_normal((mesh.num_nodes, 4))
    U[:, 3] = rng.standard_normal(mesh.num_nodes)
    return U


@pytest.mark.parametrize("again", range(4))
def test_first_adjoint_assemblies_on_one_disc(again):
    """The transposed block map is built once, by whichever thread comes first."""
    mesh = kuhn_cube(6, jitter=0.2, seed=again)

    def adjoint(d, seed):
        m = api.Mechanics(d, api.NEOHOOKEAN, [ROW])
        m.set_solution(_state(mesh, seed))
        s = api.SolInfo(d)
        return m, s, lambda: api.assemble(m, s, api.ADJOINT, jacobian=True, save_states=False)

    alone = []
    for seed in range(4):
        m, s, go = adjoint(api.Disc(mesh), seed)
        go()
        alone.append(s.dRdu_csr())
    d = api.Disc(mesh)
    kept = [adjoint(d, seed) for seed in range(4)]
    _together([k[2] for k in kept])
    for (m, s, _), A in zip(kept, alone):
        assert np.array_equal(s.dRdu_csr(), A)


def _program(n, seed, precision):
    """A discretization, an assembly and a solve of its own, as one thread's program."""
    mesh = kuhn_cube(n, jitter=0.2, seed=seed)
    d = api.Disc(mesh)
    m = api.Mechanics(d, api.J2, [ROW])
    U = _state(mesh, seed)
    U[:, 0] += 0.002 * mesh.coords[:, 0]
    m.set_solution(U)
    s = api.SolInfo(d)
    api.assemble(m, s, api.PRIMAL, jacobian=True, save_states=True)
    bcs = api.Bcs(d, [(0, "xmin", "0.0"), (1, "xmin", "0.0"), (2, "xmin", "0.0"), (0, "xmax", "0.002*t")], [])
    api.set_jac_dbcs(m, s, bcs, 1.0)
    x, st = api.solve(s, -s.R, params=api.solve_params(krylov_size=60, max_iters=20000, tolerance=1e-10,
                                                       precision=precision, inner_iters=30))
    assert st["converged"]
    return d.colors(), s.dRdu_csr(), x


@pytest.mark.parametrize("again", range(3))
def test_programs_side_by_side(again):
    """Colourings and persistent cycles, which take the whole chip each, on the
    streams of four threads."""
    jobs = [lambda n=n, p=p, k=k: _program(n, 10 * again + k, p)
            for k, (n, p) in enumerate([(12, api.MIXED), (9, api.FP64), (12, api.MIXED_F32), (10, api.NESTED_F64)])]
    alone = [j() for j in jobs]
    for a, b in zip(alone, _together(jobs)):
        assert all(np.array_equal(x, y) for x, y in zip(a, b))
