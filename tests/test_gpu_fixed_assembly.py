"""The fixed-point Jacobian assembly against the FP64 one (overwrite = 0 into
zeros), where its layouts and scales change: pinwheels whose axis edge, axis
nodes and axis rows have more terms than the gather keeps ahead; materials and
element sizes many orders of magnitude apart; undeformed, strongly deformed
and not finite states. Both sum the same element blocks, so they agree to
rounding: 1e-13 of each row's largest entry, as between the other strategies."""
import numpy as np
import pytest

from goal_gb300 import api
from goal_gb300.mesh import Mesh, graded_block, kuhn_cube, orient_positive

pytestmark = pytest.mark.gpu

J2 = [200e3, 0.3, 1000.0, 250.0, 1.0]


def _mesh(coords, tets, elem_set=None, names=("a",)):
    tets = orient_positive(coords, np.asarray(tets, np.int32))
    es = np.zeros(len(tets), np.int32) if elem_set is None else elem_set
    return Mesh(coords=coords, tets=tets, elem_set=es, elem_set_names=list(names), node_sets={}, side_sets={})


def _pinwheel(m):
    """m tets around the edge of nodes 0 and 1."""
    t = 2 * np.pi * np.arange(m) / m
    ring = np.stack([np.cos(t), np.sin(t), 0.5 + 0.1 * np.sin(3 * t)], axis=1)
    coords = np.concatenate([[[0.0, 0.0, 0.0], [0.0, 0.0, 1.0]], ring])
    return _mesh(coords, [[0, 1, 2 + i, 2 + (i + 1) % m] for i in range(m)])


def _both(mesh, model, mats, U, mode, Fp_old=None, eq=None):
    d = api.Disc(mesh)
    m = api.Mechanics(d, model, mats)
    m.set_solution(U)
    if Fp_old is not None:
        m.set_state(api.FP_OLD, Fp_old)
        m.set_state(api.EQPS_OLD, eq)
    s, z = api.SolInfo(d), api.SolInfo(d)
    api.assemble(m, s, mode, jacobian=True, save_states=False)
    api.assemble(m, z, mode, jacobian=True, save_states=False, overwrite=False)
    return d, s, z


def _close(d, s, z):
    assert np.array_equal(s.R, z.R)
    rows = d.graph()[0]
    A, B = s.dRdu_csr(), z.dRdu_csr()
    top = np.maximum.reduceat(np.abs(B), rows[:-1])
    off = np.maximum.reduceat(np.abs(A - B), rows[:-1])
    assert np.all(off <= 1e-13 * top), float((off / top).max())


def _state(mesh, scale, seed):
    rng = np.random.default_rng(seed)
    U = rng.standard_normal((mesh.num_nodes, 4))
    U[:, :3] *= scale
    return U


@pytest.mark.parametrize("mode", [api.PRIMAL, api.ADJOINT])
@pytest.mark.parametrize("m", [3, 17, 33, 61, 127])
def test_rows_longer_than_the_gather_keeps_ahead(m, mode):
    mesh = _pinwheel(m)
    _close(*_both(mesh, api.J2, [J2], _state(mesh, 2e-3 / m, 1), mode))


@pytest.mark.parametrize("model", [api.NEOHOOKEAN, api.J2])
@pytest.mark.parametrize("scale", [0.0, 1e-9, 1e-3, 0.05])
def test_deformations(model, scale):
    mesh = kuhn_cube(4, jitter=0.2, seed=2)
    rng = np.random.default_rng(4)
    S = 1e-3 * rng.standard_normal((mesh.num_elems, 3, 3))
    Fp = np.eye(3) + 0.5 * (S + S.transpose(0, 2, 1))
    old = (Fp, rng.uniform(0.0, 0.01, mesh.num_elems)) if model == api.J2 else (None, None)
    _close(*_both(mesh, model, [J2], _state(mesh, scale / 4, 3), api.PRIMAL, *old))


@pytest.mark.parametrize("mode", [api.PRIMAL, api.ADJOINT])
def test_scales_far_apart(mode):
    """Materials twelve orders of magnitude apart in neighbouring elements, and
    a part of micrometres."""
    mesh = graded_block(3000, seed=4, regions=4)
    mats = [[10.0 ** e, 0.3, 100.0, 10.0 ** (e - 3), 1.0] for e in (-3.0, 9.0, 3.0, 6.0)]
    _close(*_both(mesh, api.J2, mats, _state(mesh, 1e-5, 5), mode))
    mesh = kuhn_cube(3, length=(1e-6, 2e-6, 1e-6), jitter=0.2, seed=1)
    _close(*_both(mesh, api.NEOHOOKEAN, [J2], _state(mesh, 1e-9, 6), mode))


@pytest.mark.parametrize("mode", [api.PRIMAL, api.ADJOINT])
def test_not_a_number_stays_where_it_was(mode):
    mesh = kuhn_cube(3)
    U = _state(mesh, 1e-4, 7)
    U[10, 1] = np.nan
    d, s, z = _both(mesh, api.NEOHOOKEAN, [J2], U, mode)
    A, B = s.dRdu_csr(), z.dRdu_csr()
    assert np.isnan(B).any() and not np.isnan(B).all()
    assert np.array_equal(np.isnan(A), np.isnan(B)) and np.array_equal(np.isnan(s.R), np.isnan(z.R))


@pytest.mark.parametrize("mode", [api.PRIMAL, api.ADJOINT])
@pytest.mark.parametrize("n", [1, 2, 9, 10, 12, 26])
def test_element_counts(n, mode):
    """6 n^3 elements: four, two and one thread to an element, in blocks of 64
    and of 128, the last block ragged."""
    mesh = kuhn_cube(n, jitter=0.2, seed=n)
    _close(*_both(mesh, api.J2, [J2], _state(mesh, 2e-3 / n, 8), mode))


@pytest.mark.parametrize("model,K", [(api.NEOHOOKEAN, 1000.0), (api.J2, 1000.0), (api.J2, 0.0)])
@pytest.mark.parametrize("n,scale", [(1, 1e-9), (5, 1e-3), (5, 0.02), (21, 1e-3)])
def test_residual_alone(model, K, n, scale):
    """The residual chain and the Jacobian chain form R from different products:
    some hundred roundings of terms no larger than R's largest entries in a
    state far from equilibrium, 1e-13 of them."""
    mesh = kuhn_cube(n, jitter=0.2, seed=n)
    d = api.Disc(mesh)
    m = api.Mechanics(d, model, [[200e3, 0.3, K, 250.0, 1.0]])
    m.set_solution(_state(mesh, scale / n, 9))
    s, z = api.SolInfo(d), api.SolInfo(d)
    api.assemble(m, s, api.PRIMAL, jacobian=True, save_states=False)
    api.assemble(m, z, api.PRIMAL, jacobian=False, save_states=False)
    A, B = s.R.reshape(-1, 4), z.R.reshape(-1, 4)
    for c in (slice(0, 3), slice(3, 4)):
        assert np.abs(A[:, c] - B[:, c]).max() <= 1e-13 * np.abs(A[:, c]).max()
