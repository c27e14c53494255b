"""The work that a program built on goal_gb300 has it do, as timed cases.

A simulation with this package builds a discretization from its mesh, and then
per load step assembles Jacobians and residuals, solves the Newton systems and,
for goal-oriented adaptation, the transposed system on the refined mesh. The
cases take each of these through the public entry points (``goal_gb300.api``
and, for vectors that stay on the GPU, the C ABI's device views), from the
regression tests' few hundred tets to the 64^3 cube of the benchmark.

Materials, element counts and solver settings are those of the repository's
tests and benchmark: J2 with E = 200e3, nu = 0.3, K = 1000, Y = 250, c0 = 1 on
Kuhn cubes (interior nodes moved by up to 0.2 h), and the graded 4x1x1 block
with eight neo-Hookean material regions.
"""
import ctypes
import functools

import numpy as np
import torch

from goal_gb300 import api, lib
from goal_gb300._abi import SolveStats
from goal_gb300.mesh import Mesh, graded_block, kuhn_cube

J2_ROW = [200e3, 0.3, 1000.0, 250.0, 1.0]
RHO = 20.0  # of the KS von Mises functional
CLAMPED = [(0, "xmin", "0.0"), (1, "xmin", "0.0"), (2, "xmin", "0.0")]


def _pulled(case):
    """Clamped at x = 0, pulled along x at x = 1 by the case's displacement."""
    return CLAMPED + [(0, "xmax", "%r*t" % case.get("pull", 0.002))]


# how a solve of each precision is set up: restart length and inner iterations
PRECISION = {"fp64": api.FP64, "mixed": api.MIXED, "mixed_f32": api.MIXED_F32, "nested_f64": api.NESTED_F64}


def listed():
    return [
        # a Jacobian assembly of the size of the regression meshes: latency and launches
        {"name": "jacobian_384_tets", "kind": "assemble", "mesh": "cube", "n": 4, "model": "j2", "chain": "jacobian",
         "load": 1.0},
        # a graded part with eight material regions, neo-Hookean, odd counts
        {"name": "jacobian_graded_block", "kind": "assemble", "mesh": "block", "part": 7, "n": 16,
         "model": "nh", "chain": "jacobian", "load": 1.0},
        # the benchmark's mesh: a Newton iteration's Jacobian, half of the points plastic
        {"name": "jacobian_384k_tets", "kind": "assemble", "mesh": "cube", "n": 40, "model": "j2",
         "chain": "jacobian", "load": 1.0},
        # the transposed Jacobian and dM/du of a KS von Mises functional on a fine mesh
        {"name": "adjoint_1.5M_tets", "kind": "assemble", "mesh": "cube", "n": 63, "model": "j2", "chain": "adjoint",
         "load": 1.0},
        # a Newton iteration's second half: the residual alone
        {"name": "residual_384k_tets", "kind": "assemble", "mesh": "cube", "n": 40, "model": "j2",
         "chain": "residual", "load": 1.0},
        # small and medium Newton systems in FP64 with block-Jacobi
        {"name": "solve_fp64_2.9k_dofs", "kind": "solve", "n": 8, "precision": "fp64", "learned": False},
        {"name": "solve_fp64_20k_dofs", "kind": "solve", "n": 16, "precision": "fp64", "learned": False},
        # the nested solver with the learned preconditioner, and at the size of the fine cube without it
        {"name": "solve_learned_276k_dofs", "kind": "solve", "n": 40, "precision": "mixed", "learned": True},
        {"name": "solve_mixed_1.1M_dofs", "kind": "solve", "n": 64, "precision": "mixed", "learned": False},
        # whole calls: a load step's Newton solve, and the nested adjoint with its error indicators
        {"name": "newton_6k_tets", "kind": "newton", "n": 10, "precision": "mixed", "pull": 0.002},
        {"name": "nested_adjoint_83k_tets", "kind": "nested", "n": 12, "precision": "mixed", "pull": 0.002},
        # a new mesh, as after each adaptation: graph, colouring, element layout
        {"name": "disc_83k_tets", "kind": "disc", "mesh": "cube", "n": 24},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["assemble", "assemble", "assemble", "solve", "solve", "newton", "nested", "disc"])
    if kind in ("assemble", "disc"):
        case = {"kind": kind, "mesh": rng.choice(["cube", "cube", "block"])}
        case["n"] = _log_int(rng, 4, 63 if kind == "assemble" else 48)
        if case["mesh"] == "block":
            case["part"] = rng.randrange(1000)
        if kind == "assemble":
            case.update(model=rng.choice(["j2", "nh"]), chain=rng.choice(["jacobian", "adjoint", "residual"]),
                        load=round(rng.uniform(0.5, 1.5), 3))
        return case
    if kind == "solve":
        precision = rng.choice(["fp64", "mixed", "mixed", "mixed_f32", "nested_f64"])
        most = {"fp64": 16, "nested_f64": 40}.get(precision, 56)
        return {"kind": kind, "n": _log_int(rng, 4, most), "precision": precision,
                "learned": precision != "fp64" and rng.random() < 0.5}
    return {"kind": kind, "n": _log_int(rng, 4, 12), "precision": rng.choice(["mixed", "mixed_f32"]),
            "pull": round(rng.uniform(0.0005, 0.002), 6)}


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=4)
def _grid(n):
    return kuhn_cube(n)


def _cube(n, seed):
    """The Kuhn cube with its interior nodes moved by up to 0.2 h."""
    g = _grid(n)
    inner = np.all((g.coords > 1e-9) & (g.coords < 1.0 - 1e-9), axis=1)
    move = np.random.default_rng(seed).uniform(-0.2, 0.2, g.coords.shape) / n
    return Mesh(coords=g.coords + move * inner[:, None], tets=g.tets, elem_set=g.elem_set,
                elem_set_names=g.elem_set_names, node_sets=g.node_sets, side_sets=g.side_sets)


@functools.lru_cache(maxsize=4)
def _block(n, part):
    """A graded block of eight material regions with about the cube's element count."""
    return graded_block(6 * n ** 3, seed=part, regions=8)


def _mesh(case, seed):
    return _block(case["n"], case["part"]) if case.get("mesh") == "block" else _cube(case["n"], seed)


def _renumbered(mesh, seed):
    """The mesh with its elements listed from another one on, as another run of a mesher lists them."""
    first = seed * 7919 % mesh.num_elems
    return Mesh(coords=mesh.coords, tets=np.roll(mesh.tets, -first, axis=0), elem_set=np.roll(mesh.elem_set, -first),
                elem_set_names=mesh.elem_set_names, node_sets=mesh.node_sets, side_sets=mesh.side_sets)


def _materials(case, mesh, seed):
    rows = len(mesh.elem_set_names)
    if rows == 1:
        return np.array([J2_ROW])
    rng = np.random.default_rng(seed + 1)
    E = np.exp(rng.normal(np.log(1000.0), 0.5, rows))
    return np.stack([E, rng.uniform(0.2, 0.45, rows), np.full(rows, 100.0), rng.uniform(50.0, 300.0, rows),
                     np.ones(rows)], axis=1)


def _fields(mesh, load, seed):
    """Displacements and pressures of a bent part with some noise; for J2 a
    plastic history with which, at load 1, about half of the cube's points yield."""
    rng = np.random.default_rng(seed + 2)
    x = mesh.coords
    h = float(np.cbrt(6.0 * np.prod(x.max(axis=0) - x.min(axis=0)) / mesh.num_elems))
    U = np.empty((mesh.num_nodes, 4))
    U[:, :3] = load * 4.4e-4 * np.sin(np.pi * x) + 1e-4 * h * rng.standard_normal(x.shape)
    U[:, 3] = rng.standard_normal(mesh.num_nodes)
    S = rng.standard_normal((mesh.num_elems, 3, 3)) * 3e-4
    S = 0.5 * (S + S.transpose(0, 2, 1))
    S -= np.trace(S, axis1=1, axis2=2)[:, None, None] / 3.0 * np.eye(3)
    Fp_old = np.eye(3) + S + 0.5 * S @ S
    return U, Fp_old, rng.uniform(0.0, 0.01, mesh.num_elems)


def _loaded(mesh, seed):
    """Displacements of a load step under way: stretched along x, with noise."""
    rng = np.random.default_rng(seed + 3)
    x = mesh.coords
    h = float(np.cbrt(6.0 / mesh.num_elems))
    U = np.empty((mesh.num_nodes, 4))
    U[:, 0] = 0.002 * x[:, 0]
    U[:, 1] = -0.0007 * x[:, 1] * x[:, 0]
    U[:, 2] = -0.0007 * x[:, 2] * x[:, 0]
    U[:, :3] += 2e-4 * h * rng.standard_normal((mesh.num_nodes, 3))
    U[:, 3] = 50.0 * x[:, 0] + rng.standard_normal(mesh.num_nodes)
    return U


class _Device:
    """FP64 values at a device address that a handle of the library owns; a
    tensor made from it keeps this object, and so the handle, alive."""

    def __init__(self, owner, address, count):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (address, False), "shape": (count,), "typestr": "<f8", "version": 3}


def _on_device(owner, address, count):
    return torch.as_tensor(_Device(owner, address.value, count), device="cuda")


def _views(s):
    """R, dM/du and the 4x4 blocks of a SolInfo, in place."""
    R, M, A = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()
    api.check(lib().goal_sol_info_device_view(s.h, ctypes.byref(R), ctypes.byref(M), ctypes.byref(A)))
    return (_on_device(s, R, s.disc.num_dofs), _on_device(s, M, s.disc.num_dofs),
            _on_device(s, A, 16 * s.disc.nnzb))


def _solution_view(m):
    U = ctypes.c_void_p()
    api.check(lib().goal_mechanics_device_solution(m.h, ctypes.byref(U)))
    return _on_device(m, U, m.disc.num_dofs)


def _params(precision, learned=False, tolerance=1e-12):
    return api.solve_params(krylov_size=100, max_iters=20000, tolerance=tolerance, precision=PRECISION[precision],
                            inner_iters=60, precond=api.PRECOND_LEARNED if learned else api.PRECOND_BJ)


@functools.lru_cache(maxsize=1)
def _trained():
    """A network trained on a small cube's Newton system, as a program keeps it."""
    mesh = _cube(8, 1)
    d = api.Disc(mesh)
    m = api.Mechanics(d, api.J2, [J2_ROW])
    m.set_solution(_loaded(mesh, 1))
    s = api.SolInfo(d)
    api.assemble(m, s, api.PRIMAL, jacobian=True, save_states=True)
    api.set_jac_dbcs(m, s, api.Bcs(d, _pulled({})), 1.0)
    net = api.Learned(seed=3)
    net.train([s], epochs=60, lr=3e-3, num_probes=8, seed=5)
    return net


def prepare(case, seed):
    kind = case["kind"]
    mesh = _mesh(case, seed)
    if kind == "disc":
        return {"case": case, "mesh": _renumbered(mesh, seed)}
    d = api.Disc(mesh)
    s = api.SolInfo(d)
    state = {"case": case, "disc": d, "s": s}
    if kind == "assemble":
        m = api.Mechanics(d, api.J2 if case["model"] == "j2" else api.NEOHOOKEAN, _materials(case, mesh, seed))
        U, Fp_old, eqps_old = _fields(mesh, case["load"], seed)
        m.set_solution(U)
        if case["model"] == "j2":
            m.set_state(api.FP_OLD, Fp_old)
            m.set_state(api.EQPS_OLD, eqps_old)
        if case["chain"] == "adjoint":  # the stored stresses that the KS functional is scaled with
            api.assemble(m, s, api.PRIMAL, jacobian=False, save_states=True)
        state.update(m=m, views=_views(s))
        return state
    m = api.Mechanics(d, api.J2, [J2_ROW])
    state["m"] = m
    if kind == "solve":
        m.set_solution(_loaded(mesh, seed))
        api.assemble(m, s, api.PRIMAL, jacobian=True, save_states=True)
        api.set_jac_dbcs(m, s, api.Bcs(d, _pulled(case)), 1.0)
        if case["learned"]:
            state["net"] = _trained()
            state["net"].attach(s)
        state.update(b=-_views(s)[0], x=torch.empty(d.num_dofs, dtype=torch.float64, device="cuda"),
                     stream=torch.cuda.ExternalStream(d.stream()))
        return state
    state.update(bcs=api.Bcs(d, _pulled(case)), start=np.zeros(d.num_dofs), U=_solution_view(m))
    if kind == "nested":
        api.primal_solve(m, s, state["bcs"], 1.0, 0.0, 30, 1e-8, _params("mixed", tolerance=1e-10))
        state["adjoint"] = api.NestedAdjoint(m, _pulled(case))
    return state


# ------------------------------------------------------------------ one pass
def run(state):
    kind = state["case"]["kind"]
    if kind == "assemble":
        chain = state["case"]["chain"]
        R, M, A = state["views"]
        if chain == "adjoint":
            q = api.assemble(state["m"], state["s"], api.ADJOINT, jacobian=True, save_states=False,
                             qoi=api.QOI_KS_VM, rho=RHO)
            return {"A": A, "M": M, "R": R, "qoi": q}
        api.assemble(state["m"], state["s"], api.PRIMAL, jacobian=chain == "jacobian", save_states=True)
        return {"A": A, "R": R} if chain == "jacobian" else {"R": R}
    if kind == "solve":
        with torch.cuda.stream(state["stream"]):
            state["x"].zero_()
        p = _params(state["case"]["precision"], state["case"]["learned"])
        api.check(lib().goal_solve_device(state["s"].h, ctypes.byref(p), state["b"].data_ptr(), state["x"].data_ptr(),
                                          ctypes.byref(SolveStats())))
        return state["x"]
    if kind == "newton":
        state["m"].set_solution(state["start"])
        api.primal_solve(state["m"], state["s"], state["bcs"], 1.0, 0.0, 30, 1e-8,
                         _params(state["case"]["precision"], tolerance=1e-10))
        return state["U"]
    if kind == "nested":
        r = state["adjoint"].run(api.QOI_KS_VM, RHO, 1.0, 0.0, _params(state["case"]["precision"]))
        return {"bound": r["bound"], "error": r["base_error"], "eta": r["eta"], "qoi": r["qoi"],
                "z": state["adjoint"].z()}
    d = api.Disc(state["mesh"])
    rows, cols = d.graph()
    return {"rows": rows, "cols": cols, "colors": d.colors()}


def work(case):
    """Bytes and FP64 operations of a pass that no implementation can avoid:
    each input read once, each output written once. Elements E and nodes N of
    the Kuhn grid, about 15 blocks per node; of a solve one product with the
    matrix, of a whole call one assembly and one product."""
    n = case["n"]
    E, N = 6.0 * n ** 3, (n + 1.0) ** 3
    blocks = 15.0 * N
    system = 16 * E + 56 * N + 32 * N + 128 * blocks
    if case["kind"] == "assemble":
        states = {"j2": 232, "nh": 72}[case["model"]] * E
        if case["chain"] == "residual":
            return {"bytes": 16 * E + 88 * N + states, "flops": 400 * E}
        return {"bytes": system + states, "flops": {"j2": 1655, "nh": 1250}[case["model"]] * E}
    if case["kind"] == "solve":
        return {"bytes": 132 * blocks + 64 * N, "flops": 32 * blocks}
    if case["kind"] == "newton":
        return {"bytes": system + 232 * E + 132 * blocks, "flops": 1655 * E + 32 * blocks}
    if case["kind"] == "nested":
        return {"bytes": 8 * (system + 232 * E + 132 * blocks), "flops": 8 * (1655 * E + 32 * blocks)}
    return {"bytes": 16 * E + 4 * E + 24 * N + 64 * blocks + 16 * N + 4 * E, "flops": 0}


# ------------------------------------------------------------------ in 64 bits, without the library
def _inv3(A):
    """Inverse and determinant of 3x3 matrices by cofactors."""
    a, b, c = A[..., 0, :], A[..., 1, :], A[..., 2, :]
    cross = lambda u, v: torch.stack([u[..., 1] * v[..., 2] - u[..., 2] * v[..., 1],  # noqa: E731
                                      u[..., 2] * v[..., 0] - u[..., 0] * v[..., 2],
                                      u[..., 0] * v[..., 1] - u[..., 1] * v[..., 0]], dim=-1)
    cof = torch.stack([cross(b, c), cross(c, a), cross(a, b)], dim=-2)
    det = (a * cof[..., 0, :]).sum(-1)
    return cof.transpose(-1, -2) / det[..., None, None], det


def _element(x, G, V, h, C, eq, mat, j2, ks):
    """One element's residual (4, 4) and, with ks = (max, scale), its value of
    the KS functional, for nodal values x (4, 4) = u, p."""
    eye = torch.eye(3, dtype=x.dtype, device=x.device)
    E, nu, K, Y, c0 = (mat[i] for i in range(5))
    kappa, mu = E / (3 * (1 - 2 * nu)), E / (2 * (1 + nu))
    F = eye + x[:, :3].T @ G
    Fi, J = _inv3(F)
    p, gp = x[:, 3].mean(), x[:, 3] @ G
    B = F @ C @ F.T
    Ic = torch.trace(B)
    s = mu * J ** (-2.0 / 3.0) * (B - Ic / 3 * eye)
    mag = torch.sqrt((s * s).sum())
    if j2:
        mubar = mu * J ** (-2.0 / 3.0) * Ic / 3
        f = mag - (2.0 / 3.0) ** 0.5 * (Y + K * eq)
        s = torch.where(f > 1e-12, 1 - 2 * mubar * f / (2 * mubar + 2 * K / 3) / mag, torch.ones_like(f)) * s
    sigma = s / J + p * eye
    H = Fi.T
    g = G @ Fi  # rows F^-T grad phi_a
    Ru = V * J * g @ sigma
    tau = c0 * h * h / (2 * mu)
    Rp = V * ((p / kappa - 0.5 * (J - 1 / J)) / 4 + tau * J * (g @ (H @ gp)))
    vm = 1.5 ** 0.5 * torch.sqrt((s * s).sum()) / J
    value = torch.exp(RHO * (vm - ks[0])) * V / (RHO * ks[1])
    return torch.cat([Ru, Rp[:, None]], dim=1), value, vm


def _reference(mesh, mats, U, Fp_old, eq_old, j2, what):
    """The assembled system of ``what`` ("residual", "jacobian", "adjoint") by
    automatic differentiation of the element residual."""
    dev = "cuda"
    T = lambda a: torch.as_tensor(np.asarray(a), device=dev)  # noqa: E731
    t = T(mesh.tets.astype(np.int64))
    X = T(mesh.coords)[t]
    Ji, det = _inv3((X[:, 1:] - X[:, :1]).transpose(1, 2))
    G = torch.cat([-Ji.sum(1, keepdim=True), Ji], dim=1)
    V = det / 6
    h = torch.sqrt(sum(((X[:, a] - X[:, b]) ** 2).sum(-1) for a in range(4) for b in range(a)) / 6)
    Fpi = _inv3(T(Fp_old))[0]
    C = Fpi @ Fpi.transpose(1, 2)
    x = T(U).reshape(-1, 4)[t]
    args = [G, V, h, C, T(eq_old), T(mats)[T(mesh.elem_set.astype(np.int64))]]
    E, N = t.shape[0], mesh.num_nodes
    zero = torch.zeros(2, dtype=torch.float64, device=dev)
    scale = lambda ks: functools.partial(_element, j2=j2, ks=ks)  # noqa: E731
    step = 1 << 15
    parts = [slice(i, min(E, i + step)) for i in range(0, E, step)]
    call = lambda f, q: f(x[q], *(a[q] for a in args))  # noqa: E731
    R = torch.zeros(4 * N, dtype=torch.float64, device=dev)
    rows = (4 * t[:, :, None] + torch.arange(4, device=dev)).reshape(E, 16)
    vm = torch.empty(E, dtype=torch.float64, device=dev)
    for q in parts:
        r, _, vm[q] = call(torch.func.vmap(scale(zero + 1)), q)
        R.index_add_(0, rows[q].reshape(-1), r.reshape(-1))
    out = {"R": R}
    if what == "residual":
        return out
    ks = zero + 1
    if what == "adjoint":
        top = vm.max()
        ks = torch.stack([top, (torch.exp(RHO * (vm - top)) * V).sum()])
        out["qoi"] = float(top + torch.log(ks[1]) / RHO)
        out["M"] = torch.zeros_like(R)
    keys = t[:, :, None] * N + t[:, None, :]
    graph = torch.unique(keys)
    A = torch.zeros(16 * graph.numel(), dtype=torch.float64, device=dev)
    at = torch.arange(16, device=dev)
    for q in parts:
        K, M, _ = call(torch.func.vmap(torch.func.jacfwd(scale(ks))), q)
        K = K.permute(0, 1, 3, 2, 4)  # [e, a, b, i, k]
        if what == "adjoint":
            K = K.permute(0, 2, 1, 4, 3)
            out["M"].index_add_(0, rows[q].reshape(-1), M.reshape(-1))
        place = 16 * torch.searchsorted(graph, keys[q])[..., None] + at
        A.index_add_(0, place.reshape(-1), K.reshape(-1))
    out["A"], out["graph"] = A, graph
    return out


def _constrained(mesh, sys, U, case):
    """Dense matrix and right-hand side of a Newton system under _pulled."""
    N = mesh.num_nodes
    A = torch.zeros(4 * N, 4 * N, dtype=torch.float64, device="cuda")
    i, j = sys["graph"] // N, sys["graph"] % N
    at = torch.arange(4, device="cuda")
    A[4 * i[:, None, None] + at[None, :, None], 4 * j[:, None, None] + at[None, None, :]] = sys["A"].reshape(-1, 4, 4)
    R = sys["R"].clone()
    u = torch.as_tensor(U, device="cuda").reshape(-1)
    for eq, name, text in _pulled(case):
        dofs = 4 * torch.as_tensor(mesh.node_sets[name].astype(np.int64), device="cuda") + eq
        A[dofs] = 0
        A[dofs, dofs] = 1
        R[dofs] = u[dofs] - (case.get("pull", 0.002) if "t" in text else 0.0)
    return A, R


def exact(case, seed):
    mesh = _mesh(case, seed)
    if case["kind"] == "assemble":
        j2 = case["model"] == "j2"
        U, Fp_old, eqps_old = _fields(mesh, case["load"], seed)
        if not j2:
            Fp_old = np.broadcast_to(np.eye(3), Fp_old.shape).copy()
        out = _reference(mesh, _materials(case, mesh, seed), U, Fp_old, eqps_old, j2, case["chain"])
        out.pop("graph", None)
        return out
    if case["kind"] not in ("solve", "newton") or case["n"] > 10:
        return None  # no dense factorization of that size in a few seconds
    fresh = np.broadcast_to(np.eye(3), (mesh.num_elems, 3, 3)).copy()
    old = np.zeros(mesh.num_elems)

    def system(U):
        return _constrained(mesh, _reference(mesh, [J2_ROW], U, fresh, old, True, "jacobian"), U, case)

    if case["kind"] == "solve":
        A, R = system(_loaded(mesh, seed))
        return torch.linalg.solve(A, -R)
    U = np.zeros(4 * mesh.num_nodes)
    for _ in range(30):
        A, R = system(U)
        if float(R.norm()) < 1e-9:
            break
        U = U + torch.linalg.solve(A, -R).cpu().numpy()
    return torch.as_tensor(U, device="cuda")
