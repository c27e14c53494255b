"""The fixed-point Jacobian assembly over the whole range of deformations and
element shapes: its error against element blocks formed in extended precision
(80 or 113 bits, as the host has them) beside that of the FP64 assembly
(overwrite = 0 into zeros), and the elements that it leaves to FP64.

The bound: both paths share the FP64 evaluation of the integration point, and
what the fixed-point path adds is a few units of 2^-57 of a block's largest
entry, so its largest error over the mesh is that of the FP64 path but for the
chance of single roundings: 2 times it, and 8 units of FP64's rounding (1.8e-15)
where the FP64 path happens to be exact."""
import numpy as np
import pytest

from goal_gb300 import api
from goal_gb300.mesh import Mesh, kuhn_cube, orient_positive

pytestmark = pytest.mark.gpu

ROW = [200e3, 0.3, 1000.0, 250.0, 1.0]
X = np.longdouble


def _blocks(mesh, model, U, Fp_old, eq):
    """The element blocks K (E, 4, 4, 4, 4) [e, a, b, row, column] by the formulas at
    the head of element.cu."""
    E_, nu, K, Y, c0 = (X(v) for v in ROW)
    kappa, mu = E_ / (3 * (1 - 2 * nu)), E_ / (2 * (1 + nu))
    x = mesh.coords.astype(X)[mesh.tets]
    D = np.swapaxes(x[:, 1:] - x[:, :1], 1, 2)

    def cof3(A):
        r = np.empty_like(A)
        for i in range(3):
            for j in range(3):
                a, b, c, d = (i + 1) % 3, (i + 2) % 3, (j + 1) % 3, (j + 2) % 3
                r[:, i, j] = A[:, a, c] * A[:, b, d] - A[:, a, d] * A[:, b, c]
        return r

    cd = cof3(D)
    det = (D[:, 0] * cd[:, 0]).sum(-1)
    g = np.swapaxes(cd / det[:, None, None], 1, 2)  # grad phi_1..3
    G = np.concatenate([-g.sum(1, keepdims=True), g], axis=1)
    V = det / 6
    h2 = sum(((x[:, a] - x[:, b]) ** 2).sum(-1) for a in range(4) for b in range(a)) / 6
    u = U.astype(X).reshape(-1, 4)[mesh.tets]
    mm = lambda A, B: np.einsum("eij,ejk->eik", A, B)  # noqa: E731
    eye = np.eye(3, dtype=X)
    F = eye + np.einsum("eai,eaj->eij", u[..., :3], G)
    p, gp = u[..., 3].sum(1) / 4, np.einsum("ea,eaj->ej", u[..., 3], G)
    cf = cof3(F)
    J = (F[:, 0] * cf[:, 0]).sum(-1)
    H = cf / J[:, None, None]
    C = np.broadcast_to(eye, F.shape)
    if model == api.J2:
        Fp = Fp_old.astype(X)
        ci = cof3(Fp)
        Fi = np.swapaxes(ci / (Fp[:, 0] * ci[:, 0]).sum(-1)[:, None, None], 1, 2)
        C = mm(Fi, np.swapaxes(Fi, 1, 2))
    FC = mm(F, C)
    B = mm(FC, np.swapaxes(F, 1, 2))
    Ic3 = np.trace(B, axis1=1, axis2=2) / 3
    alpha = mu * J ** (X(-2) / 3)
    s = alpha[:, None, None] * (B - Ic3[:, None, None] * eye)
    smag = np.sqrt((s * s).sum((1, 2)))
    gamma, A1, A2 = np.ones_like(J), np.zeros_like(J), np.zeros_like(J)
    if model == api.J2:
        mubar, k0 = alpha * Ic3, np.sqrt(X(2) / 3) * (Y + K * eq.astype(X))
        f = smag - k0
        at = f > 1e-12
        kh = 2 * K / 3
        c = 2 * mubar + kh
        gamma[at] = (1 - 2 * mubar * f / c / smag)[at]
        A1[at] = (2 * f * kh / (c * c * smag))[at]
        A2[at] = (2 * mubar * k0 / (c * smag * smag))[at]
    w1 = lambda v: v[:, None, None]  # noqa: E731
    ga, pJ, tJ = gamma * alpha, p * J, c0 * h2 / (2 * mu) * J
    h, m = np.einsum("eij,eaj->eai", H, G), np.einsum("eij,eaj->eai", FC, G)
    q = m - w1(Ic3) * h
    nrm = np.where(smag > 0, smag, 1)
    n = np.einsum("eij,eaj->eai", s, m)
    Xb = w1(-2 * ga / 3) * m + w1(pJ) * h
    dg = -w1(A1 * 2 * alpha / 3) * q - w1(A2) * (w1(-2 * smag / 3) * h + w1(2 * alpha / nrm) * n)
    Yb = w1(-2 * ga / 3) * h + w1(alpha) * dg
    Z = w1(ga * Ic3 - pJ) * h
    cab = np.einsum("eai,eij,ebj->eab", G, C, G)
    eab = np.einsum("eai,ebi->eab", h, h)
    v = np.einsum("eij,ej->ei", H, gp)
    w = np.einsum("ei,eai->ea", v, h)
    out = np.empty((len(J), 4, 4, 4, 4), X)
    out[..., :3, :3] = (np.einsum("eai,ebk->eabik", h, Xb) + np.einsum("eai,ebk->eabik", q, Yb) +
                        np.einsum("ebi,eak->eabik", h, Z) + (w1(ga) * cab)[..., None, None] * eye)
    out[..., :3, 3] = (w1(J) / 4 * h)[:, :, None, :]
    tw = tJ[:, None] * w
    out[..., 3, :3] = ((tw - ((J + 1 / J) / 8)[:, None])[:, :, None, None] * h[:, None] -
                       (w1(tJ) * eab)[..., None] * v[:, None, None] - tw[:, None, :, None] * h[:, :, None])
    out[..., 3, 3] = 1 / (16 * kappa) + w1(tJ) * eab
    return out * V[:, None, None, None, None]


def _kinds():
    return {"uu": (slice(0, 3), slice(0, 3)), "up": (slice(0, 3), slice(3, 4)), "pu": (slice(3, 4), slice(0, 3)),
            "pp": (slice(3, 4), slice(3, 4))}


def _graph(d):
    """Block rows and columns of the matrix's 4x4 blocks."""
    rp, ci = d.graph()
    cols = [ci[rp[4 * n]:rp[4 * n + 1]:4] // 4 for n in range(d.num_nodes)]
    rows = np.repeat(np.arange(d.num_nodes), [len(c) for c in cols])
    return rows, np.concatenate(cols)


def _as_blocks(d, vals):
    rp = d.graph()[0]
    return np.concatenate([vals[rp[4 * n]:rp[4 * n + 4]].reshape(4, -1, 4).transpose(1, 0, 2)
                           for n in range(d.num_nodes)])


def _history(mesh, model, seed=4):
    rng = np.random.default_rng(seed)
    S = 1e-3 * rng.standard_normal((mesh.num_elems, 3, 3))
    return np.eye(3) + 0.5 * (S + S.transpose(0, 2, 1)), rng.uniform(0.0, 0.01, mesh.num_elems)


def _both(mesh, model, U, mode=api.PRIMAL, **chain):
    Fp, eq = _history(mesh, model)
    d = api.Disc(mesh)
    m = api.Mechanics(d, model, [ROW])
    m.set_solution(U)
    if model == api.J2:
        m.set_state(api.FP_OLD, Fp)
        m.set_state(api.EQPS_OLD, eq)
    s, z = api.SolInfo(d), api.SolInfo(d)
    api.assemble(m, s, mode, jacobian=True, save_states=False, **chain)
    api.assemble(m, z, mode, jacobian=True, save_states=False, overwrite=False, **chain)
    return d, s, z, Fp, eq


def _deformed(mesh, F, noise, seed=3):
    rng = np.random.default_rng(seed)
    U = np.empty((mesh.num_nodes, 4))
    U[:, :3] = mesh.coords @ (np.asarray(F, float) - np.eye(3)).T + noise * rng.standard_normal((mesh.num_nodes, 3))
    U[:, 3] = 50.0 * rng.standard_normal(mesh.num_nodes)
    return U


def _flattened(n, by):
    m = kuhn_cube(n, jitter=0.2, seed=2)
    return Mesh(coords=m.coords * np.array([1.0, 1.0, by]), tets=m.tets, elem_set=m.elem_set,
                elem_set_names=m.elem_set_names, node_sets={}, side_sets={})


STATES = {"strain 1e-6": (np.eye(3), 1e-6), "strain 0.1": (np.eye(3), 0.02)}
STATES.update({f"dilation {l:g}": (l * np.eye(3), 0.005 * l) for l in (0.01, 0.1, 0.25, 2.0, 4.0, 8.0, 100.0, 1e4)})
STATES.update({f"stretch {l:g}": (np.diag([l, l ** -0.5, l ** -0.5]), 1e-3) for l in (0.25, 2.0, 5.0, 10.0, 100.0)})
STATES.update({f"shear {g:g}": (np.eye(3) + g * np.eye(3, k=1), 1e-3) for g in (1.0, 3.0, 10.0)})
STATES["shear 10"] = (np.eye(3) + 10.0 * np.eye(3, k=1), 1e-4)  # 1e-3 inverts elements


@pytest.mark.parametrize("model", [api.NEOHOOKEAN, api.J2])
@pytest.mark.parametrize("state", sorted(STATES))
def test_error_is_that_of_fp64(state, model):
    mesh = kuhn_cube(3, jitter=0.2, seed=2)
    F, noise = STATES[state]
    U = _deformed(mesh, F, noise)
    d, s, z, Fp, eq = _both(mesh, model, U)
    rows, cols = _graph(d)
    K = _blocks(mesh, model, U, Fp, eq)
    assert np.isfinite(K).all()
    ref = np.zeros((len(rows), 4, 4), X)
    place = {rc: k for k, rc in enumerate(zip(rows, cols))}
    for e, t in enumerate(mesh.tets):
        for a in range(4):
            for b in range(4):
                ref[place[t[a], t[b]]] += K[e, a, b]
    A, B = _as_blocks(d, s.dRdu_csr()), _as_blocks(d, z.dRdu_csr())
    for kind, (i, k) in _kinds().items():
        # relative to the largest entry of the kind in the block's row
        top = np.zeros(d.num_nodes, X)
        np.maximum.at(top, rows, np.abs(ref[:, i, k]).max((1, 2)))
        err = lambda M: float((np.abs(M[:, i, k] - ref[:, i, k]).max((1, 2)) / top[rows]).max())  # noqa: E731
        assert err(A) <= 2.0 * err(B) + 8 * 2.0 ** -52, (kind, err(A), err(B))


def _stretched_flat(n, mode, model):
    """Elements that an almost homogeneous deformation flattens to a ten-thousandth."""
    mesh = kuhn_cube(n, jitter=0.2, seed=2)
    return _both(mesh, model, _deformed(mesh, np.diag([1.0, 1.0, 1e-4]), 1e-8 / n), mode)


@pytest.mark.parametrize("mode", [api.PRIMAL, api.ADJOINT])
@pytest.mark.parametrize("flat", ["mesh", "state"])
@pytest.mark.parametrize("n", [1, 3, 10, 12, 26])
def test_flat_elements_are_left_to_fp64(n, flat, mode):
    """Elements flattened along z to a ten-thousandth (in the mesh; or by the
    state, then with four, two and one thread each). The entries that couple x
    and y are 1e-8 of a block's largest, and some ten roundings of terms not much
    larger than they are: 1e-12 of the largest of them, where 2^-59 of the
    block's largest entry would be 1.7e-10."""
    if flat == "mesh":
        mesh = _flattened(n, 1e-4)
        d, s, z, _, _ = _both(mesh, api.NEOHOOKEAN, _deformed(mesh, np.eye(3), 1e-8 / n), mode)
    else:
        d, s, z, _, _ = _stretched_flat(n, mode, api.NEOHOOKEAN)
    rows, cols = _graph(d)
    off = rows != cols
    A, B = _as_blocks(d, s.dRdu_csr()), _as_blocks(d, z.dRdu_csr())
    assert np.array_equal(s.R, z.R)
    assert np.abs(A - B).max() <= 1e-13 * np.abs(B).max()
    for i, k in ((0, 1), (1, 0)):
        assert np.abs(A - B)[off, i, k].max() <= 1e-12 * np.abs(B[off, i, k]).max()


@pytest.mark.parametrize("mode", [api.PRIMAL, api.ADJOINT])
@pytest.mark.parametrize("m", [3, 17, 33, 127])
def test_long_rows_in_fp64(m, mode):
    """A pinwheel of m tets around an edge, flattened by the state: rows with more
    blocks than a warp has lanes and more terms than the gather keeps ahead."""
    t = 2 * np.pi * np.arange(m) / m
    ring = np.stack([np.cos(t), np.sin(t), 0.5 + 0.1 * np.sin(3 * t)], axis=1)
    coords = np.concatenate([[[0.0, 0.0, 0.0], [0.0, 0.0, 1.0]], ring])
    tets = orient_positive(coords, np.array([[0, 1, 2 + i, 2 + (i + 1) % m] for i in range(m)], np.int32))
    mesh = Mesh(coords=coords, tets=tets, elem_set=np.zeros(m, np.int32), elem_set_names=["a"], node_sets={},
                side_sets={})
    U = _deformed(mesh, np.diag([1.0, 1.0, 1e-4]), 1e-8 / m)
    d, s, z, _, _ = _both(mesh, api.NEOHOOKEAN, U, mode)
    # the terms of each row, which cancel in some: a sum of up to m element blocks, each of some
    # ten roundings, and on the diagonal the sum of the row
    K = np.abs(_blocks(mesh, api.NEOHOOKEAN, U, None, None)).astype(float)
    terms = np.zeros((d.num_nodes, 4))
    for a in range(4):
        np.add.at(terms, mesh.tets[:, a], K[:, a].sum((1, 3)) if mode == api.PRIMAL else K[:, :, a].sum((1, 2)))
    off = np.abs(s.dRdu_csr() - z.dRdu_csr())
    rp = d.graph()[0]
    assert np.all(np.maximum.reduceat(off, rp[:-1]) <= (m + 16) * 2.0 ** -52 * terms.ravel())
    assert np.array_equal(s.R, z.R)


@pytest.mark.parametrize("mode", [api.PRIMAL, api.ADJOINT])
def test_one_flat_element_among_others(mode):
    """Rows that mix FP64 and fixed-point records, with dM/du of the KS functional."""
    mesh = kuhn_cube(4)
    c = mesh.coords.copy()
    t = mesh.tets[mesh.num_elems // 2]
    c[t[3]] += 0.998 * (c[t[:3]].mean(axis=0) - c[t[3]])
    mesh = Mesh(coords=c, tets=mesh.tets, elem_set=mesh.elem_set, elem_set_names=mesh.elem_set_names, node_sets={},
                side_sets={})
    mesh.tets = orient_positive(c, mesh.tets)
    U = _deformed(mesh, np.eye(3), 1e-6)
    d = api.Disc(mesh)
    m = api.Mechanics(d, api.NEOHOOKEAN, [ROW])
    m.set_solution(U)
    api.assemble(m, api.SolInfo(d), api.PRIMAL, jacobian=False, save_states=True)
    s, z = api.SolInfo(d), api.SolInfo(d)
    for o, over in ((s, True), (z, False)):
        api.assemble(m, o, mode, jacobian=True, save_states=False, overwrite=over, qoi=api.QOI_KS_VM, rho=1e-4)
    A, B = s.dRdu_csr(), z.dRdu_csr()
    rp = d.graph()[0]
    top = np.maximum.reduceat(np.abs(B), rp[:-1])
    assert np.all(np.maximum.reduceat(np.abs(A - B), rp[:-1]) <= 1e-13 * top)
    assert np.abs(s.dMdu - z.dMdu).max() <= 1e-13 * np.abs(z.dMdu).max()


@pytest.mark.parametrize("mode", [api.PRIMAL, api.ADJOINT])
@pytest.mark.parametrize("n", [3, 10, 12])
def test_infinities_stay_infinities(n, mode):
    """An infinite pressure reaches K^uu and K^pu of its elements, entry by entry,
    and leaves K^up and K^pp finite."""
    mesh = kuhn_cube(n, jitter=0.2, seed=1)
    U = _deformed(mesh, np.eye(3), 1e-4 / n)
    U[mesh.num_nodes // 2, 3] = np.inf
    d, s, z, _, _ = _both(mesh, api.NEOHOOKEAN, U, mode)
    rows, cols = _graph(d)
    A, B = _as_blocks(d, s.dRdu_csr()), _as_blocks(d, z.dRdu_csr())
    off = rows != cols
    assert np.isinf(B[off]).any() and np.isfinite(B[off]).any()
    assert np.array_equal(np.isfinite(A[off]), np.isfinite(B[off]))
    assert np.array_equal(np.isinf(A[off]), np.isinf(B[off]))
    assert np.array_equal(np.isnan(s.R), np.isnan(z.R)) and np.array_equal(np.isinf(s.R), np.isinf(z.R))
