"""The calls that are timed: what a program that uses this library makes it do.

Every case goes through the public Python entry points of the package (thin
ctypes calls into the C ABI).  The mesh hierarchy of a case (numbering, CSR
patterns) is built once and shared, as it is in a program that solves on one
mesh; everything that differs from call to call (convection field, forcing,
viscosity-dependent values, network weights, vectors) is made from the seed.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from to_merge_master_parmoon_gb300 import OseenProblem, PmSolver
from to_merge_master_parmoon_gb300.learned import Mlp
from to_merge_master_parmoon_gb300.solver import PmFusedSolver

MAXIT = 100
OFFDIAG = (1, 2, 3, 5, 6, 7)


def listed():
    return [
        # a small steady Oseen solve (8^3 cells): the call where latency and
        # launches count, e.g. inside a parameter study on a coarse mesh
        dict(name="solve_8_mixed", kind="solve", levels=3, nx0=2, ny0=2, nz0=2, precision="mixed",
             blocks=9, nu=1e-2, rtol=1e-10),
        # the steady 16^3 problem of the plain method, FP64 to 1e-10
        dict(name="solve_16_fp64", kind="solve", levels=4, nx0=2, ny0=2, nz0=2, precision="fp64",
             blocks=9, nu=1e-2, rtol=1e-10),
        # an ordinary steady solve, 32^3 cells, with the convection stronger
        # against the viscosity (more iterations)
        dict(name="solve_32_mixed", kind="solve", levels=5, nx0=2, ny0=2, nz0=2, precision="mixed",
             blocks=9, nu=5e-3, rtol=1e-8),
        # the same size in plain FP64
        dict(name="solve_32_fp64", kind="solve", levels=5, nx0=2, ny0=2, nz0=2, precision="fp64",
             blocks=9, nu=1e-2, rtol=1e-8),
        # the largest: the 64^3 headline problem (7.5 M unknowns), mixed precision
        dict(name="solve_64_mixed", kind="solve", levels=6, nx0=2, ny0=2, nz0=2, precision="mixed",
             blocks=1, nu=1e-2, rtol=1e-8),
        # one Crank-Nicolson step of the channel (divergence constraint scaled
        # by the step): coarse convection, assembly of every level,
        # refactorisation, right-hand side and solve
        dict(name="channel_step_mixed", kind="step", levels=4, nx0=4, ny0=4, nz0=2,
             precision="mixed", nu=1.0 / 180.0),
        # drop-in use behind an outer iteration that assembles on the host a
        # system with coupled velocity blocks (a rotating frame): upload of
        # every level's matrices, refactorisation (85x85 LU) and solve
        dict(name="update_solve_16", kind="update", levels=4, nx0=2, ny0=2, nz0=2,
             precision="mixed", nu=1e-2, rtol=1e-8),
        # a batch of independent small systems in one stacked hierarchy
        dict(name="batch_12x8", kind="batch", levels=3, systems=12, precision="mixed", rtol=1e-8),
        # tetrahedral mesh (6 tetrahedra per cube)
        dict(name="tetra_8_mixed", kind="tetra", levels=3, precision="mixed", nu=1e-2, rtol=1e-8),
        # the smoother alone, called as a level operator on host vectors
        dict(name="vanka_16_fp64", kind="vanka", levels=4, nx0=2, ny0=2, nz0=2, nu=1e-2, sweeps=2),
        # the coupled defect alone, called as a level operator on host vectors
        dict(name="defect_32_fp64", kind="defect", levels=5, nx0=2, ny0=2, nz0=2, nu=1e-2),
        # a mini-batch of the learned smoother's training: forward, loss, backward
        dict(name="mlp_gradient_4096", kind="mlp", rows=4096),
    ]


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "step", "update", "batch", "tetra", "vanka",
                       "defect", "mlp"])
    logu = lambda lo, hi: float(10 ** rng.uniform(math.log10(lo), math.log10(hi)))  # noqa: E731
    if kind == "mlp":
        return dict(kind=kind, rows=int(logu(64, 8192)))
    if kind == "batch":
        return dict(kind=kind, levels=rng.choice([2, 3, 4]), systems=rng.randint(2, 12),
                    precision=rng.choice(["mixed", "fp64"]), rtol=logu(1e-9, 1e-6))
    if kind == "tetra":
        return dict(kind=kind, levels=rng.choice([2, 3]), precision=rng.choice(["mixed", "fp64"]),
                    nu=logu(1e-2, 1e-1), rtol=logu(1e-9, 1e-6))
    levels = rng.choice([2, 3, 4] if kind == "update" else [2, 3, 4, 5])
    top = 3 if levels < 5 else 2
    n0 = dict(levels=levels, nx0=rng.randint(1, top), ny0=rng.randint(1, top),
              nz0=rng.randint(1, top))
    if kind == "step":
        n0 = dict(levels=min(levels, 4), nx0=rng.choice([2, 4]), ny0=rng.randint(2, 4),
                  nz0=2)  # periodic directions need an even number
        return dict(kind=kind, precision=rng.choice(["mixed", "mixed", "fp64"]),
                    nu=logu(1.0 / 180.0, 2e-2), **n0)
    out = dict(kind=kind, nu=logu(5e-3, 1e-1), **n0)
    if kind == "vanka":
        return dict(sweeps=rng.randint(1, 4), **out)
    if kind == "defect":
        return out
    out.update(precision=rng.choice(["mixed", "mixed", "fp64"]), rtol=logu(1e-10, 1e-6))
    if kind == "solve":
        out["blocks"] = rng.choice([1, 9])
    return out


# ------------------------------------------------------------------ inputs --
@functools.lru_cache(maxsize=4)
def _mesh(levels, nx0, ny0, nz0):
    """Hierarchy on a box of cubic cells; its values are replaced."""
    return OseenProblem(n_levels=levels, nu=1e-2, seed=0, nx0=nx0, ny0=ny0, nz0=nz0,
                        box=(0.0, 0.5 * nx0, 0.0, 0.5 * ny0, 0.0, 0.5 * nz0))


@functools.lru_cache(maxsize=2)
def _one_block(levels, nx0, ny0, nz0):
    return _mesh(levels, nx0, ny0, nz0).descs_one_block()


@functools.lru_cache(maxsize=2)
def _channel(levels, nx0, ny0, nz0):
    P = OseenProblem(n_levels=levels, nu=1.0 / 180.0, seed=0, example="channel", nx0=nx0, ny0=ny0,
                     nz0=nz0, box=(0.0, 2 * np.pi, -1.0, 1.0, 0.0, np.pi), periodic="xz",
                     stretch_y=2.5, perturb=0.05)
    return P, P.descs_one_block()


def _mesh_key(case):
    return case["levels"], case["nx0"], case["ny0"], case["nz0"]


def _cells(case, level):
    """Cells per direction, node coordinates [nu, 3] and cell maps of a level."""
    P = _mesh(*_mesh_key(case))
    n = [case[k] << level for k in ("nx0", "ny0", "nz0")]
    h = 0.5 / (1 << level)
    ud = torch.from_numpy(P.arrays(level)["cell_udofs"].astype(np.int64)).cuda()
    c = torch.arange(ud.shape[0], device="cuda")
    org = torch.stack([c % n[0], (c // n[0]) % n[1], c // (n[0] * n[1])], 1).double()
    k = torch.arange(27, device="cuda")
    loc = torch.stack([k % 3, (k // 3) % 3, k // 9], 1).double()
    xyz = torch.empty((P.desc(level).n_udof, 3), dtype=torch.float64, device="cuda")
    xyz[ud] = h * (org[:, None, :] + 0.5 * loc[None])
    return h, xyz, ud


def _modes(rng, count=8):
    return rng.integers(1, 5, (count, 3)).astype(float), rng.standard_normal((count, 3)), \
        rng.uniform(0, 2 * np.pi, count)


def _convection(modes, xyz, scale):
    """Divergence-free Fourier field [b1|b2|b3]: sum of curls a sin(2 pi k.x + phi)."""
    b = torch.zeros_like(xyz)
    for k, a, phi in zip(*modes):
        c = 2 * np.pi * torch.cos(2 * np.pi * (xyz @ torch.tensor(k, device="cuda")) + phi)
        b += c[:, None] * torch.tensor(np.cross(k, a), device="cuda")
    return b.T.contiguous().reshape(-1) * scale


def _field_scale(modes, xyz):
    b = _convection(modes, xyz, 1.0).reshape(3, -1)
    return 1.0 / float(b.square().sum(0).sqrt().max())


def _load(modes, case):
    """Load vector of a smooth seeded forcing on the finest level (u = 0 walls)."""
    P = _mesh(*_mesh_key(case))
    h, xyz, ud = _cells(case, case["levels"] - 1)
    f = torch.zeros_like(xyz)
    for k, a, phi in zip(*modes):
        s = torch.sin(2 * np.pi * (xyz @ torch.tensor(k, device="cuda")) + phi)
        f += s[:, None] * torch.tensor(a, device="cuda")
    m = torch.tensor([[4.0, 2, -1], [2, 16, 2], [-1, 2, 4]], dtype=torch.float64,
                     device="cuda") * (h / 30)
    M = torch.kron(m, torch.kron(m, m))
    d = P.desc(P.n_levels - 1)
    b = torch.zeros(3 * d.n_udof + d.n_pdof, dtype=torch.float64, device="cuda")
    for c in range(3):
        part = torch.zeros(d.n_udof, dtype=torch.float64, device="cuda")
        part.index_put_((ud.reshape(-1),), (f[:, c][ud] @ M).reshape(-1), accumulate=True)
        part[d.n_active:] = 0
        b[c * d.n_udof:(c + 1) * d.n_udof] = torch.round(part, decimals=12)
    return b


def _steady(case, seed):
    """Seeded convection on every level and load vector of the finest."""
    rng = np.random.default_rng(seed)
    bm, fm = _modes(rng), _modes(rng)
    xyz = [_cells(case, lev)[1] for lev in range(case["levels"])]
    scale = _field_scale(bm, xyz[-1])
    return [_convection(bm, x, scale) for x in xyz], _load(fm, case)


def _assembled(case, conv, descs, **options):
    """A set-up handle with this convection field assembled on every level."""
    P = _mesh(*_mesh_key(case))
    S = PmSolver(descs, **options)
    for lev in range(P.n_levels):
        hh = torch.from_numpy(P.cell_sizes(lev)).cuda()
        torch.cuda.synchronize()
        S.assemble_level_device(lev, hh.data_ptr(), conv[lev].data_ptr(), case["nu"])
    S.refactor()
    return S


def _keys(rowptr, col, n):
    rp = torch.from_numpy(rowptr.astype(np.int64)).cuda()
    rows = torch.repeat_interleave(torch.arange(rp.numel() - 1, device="cuda"), rp.diff())
    return rows * n + torch.from_numpy(col.astype(np.int64)).cuda()


def _gradients(h):
    """Q2 gradient products of a cube of edge h: G[i][j] = int d_i phi_a d_j phi_b,
    and quadrature tables phi [64, 27], dphi [64, 27, 3], w [64], ref. points."""
    t, w1 = np.polynomial.legendre.leggauss(4)
    v = np.stack([0.5 * t * (t - 1), 1 - t * t, 0.5 * t * (t + 1)], 1)
    d = np.stack([t - 0.5, -2 * t, t + 0.5], 1)
    # order: quadrature z, y, x; local a + 3 b + 9 c
    flat = lambda x, y, z: np.einsum("pa,qb,rc->rqpcba", x, y, z).reshape(64, 27)  # noqa: E731
    phi = flat(v, v, v)
    dphi = np.stack([flat(d, v, v), flat(v, d, v), flat(v, v, d)], 2) * (2 / h)
    w = np.einsum("r,q,p->rqp", w1, w1, w1).reshape(64) * (h / 2) ** 3
    pts = np.stack([np.tile(t, 16), np.tile(np.repeat(t, 4), 4), np.repeat(t, 16)], 1)
    T = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    phi, dphi, w, pts = T(phi), T(dphi), T(w), T(pts)
    G = torch.einsum("q,qai,qbj->ijab", w, dphi, dphi)
    return G, phi, dphi, w, pts


def _rotating_frame(P, rate):
    """Coriolis term 2 rate (e_z x u, v) on every level of P, in its host
    arrays: A12 -= 2 rate M, A21 += 2 rate M with the mass matrix M."""
    for lev in range(P.n_levels):
        a = P.arrays(lev)
        nu = a["n_udof"]
        _, phi, _, w, _ = _gradients(0.5 / (1 << lev))
        M = torch.einsum("q,qa,qb->ab", w, phi, phi)
        ud = torch.from_numpy(a["cell_udofs"].astype(np.int64)).cuda()
        keys = _keys(a["a_rowptr"], a["a_col"], nu)
        want = (ud[:, :, None] * nu + ud[:, None, :]).reshape(-1)
        pos = torch.searchsorted(keys, want).clamp_(max=keys.numel() - 1)
        ok = (keys[pos] == want) & \
             (ud < a["n_active"])[:, :, None].expand(-1, -1, 27).reshape(-1)
        mass = torch.zeros(keys.numel(), dtype=torch.float64, device="cuda")
        mass.index_put_((pos[ok],), M.expand(ud.shape[0], 27, 27).reshape(-1)[ok],
                        accumulate=True)
        mass = np.round(mass.cpu().numpy(), 14)
        a["a"][1] -= 2 * rate * mass
        a["a"][3] += 2 * rate * mass


def _options(case, norm):
    return dict(precision=case["precision"], restart=20, maxit=MAXIT,
                res_norm_min=case["rtol"] * norm)


def _state_vector(case, seed):
    """A rough iterate on the finest level that meets u = 0 on the walls."""
    d = _mesh(*_mesh_key(case)).desc(case["levels"] - 1)
    u = np.random.default_rng(seed + 1).standard_normal(3 * d.n_udof + d.n_pdof) * 0.1
    for k in range(3):
        u[k * d.n_udof + d.n_active:(k + 1) * d.n_udof] = 0.0
    return u


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind == "mlp":
        net = Mlp(seed=int(seed) % 1000, max_batch=max(case["rows"], 128))
        g = torch.Generator(device="cuda").manual_seed(int(seed))
        X = torch.randn(case["rows"], 397, device="cuda", generator=g)
        T = torch.randn(case["rows"], 85, device="cuda", generator=g)
        return dict(kind=kind, net=net, X=X, T=T)
    if kind == "solve":
        conv, b = _steady(case, seed)
        key = _mesh_key(case)
        descs = _one_block(*key) if case["blocks"] == 1 else _mesh(*key).descs
        S = _assembled(case, conv, descs, **_options(case, float(b.norm())))
        return dict(kind=kind, S=S, b=b, x=torch.zeros_like(b),
                    n3=3 * _mesh(*key).desc(case["levels"] - 1).n_udof)
    if kind in ("vanka", "defect"):
        conv, b = _steady(case, seed)
        S = _assembled(case, conv, _mesh(*_mesh_key(case)).descs, precision="fp64")
        u = _state_vector(case, seed)
        return dict(kind=kind, S=S, u=u, b=b.cpu().numpy(), level=case["levels"] - 1,
                    sweeps=case.get("sweeps", 0))
    if kind == "update":
        P = OseenProblem(n_levels=case["levels"], nu=case["nu"], seed=int(seed) % 100000,
                         nx0=case["nx0"], ny0=case["ny0"], nz0=case["nz0"],
                         box=(0.0, 0.5 * case["nx0"], 0.0, 0.5 * case["ny0"], 0.0,
                              0.5 * case["nz0"]))
        b = P.rhs()
        _rotating_frame(P, float(rng.uniform(0.2, 0.5)))
        S = PmSolver(P.descs, **_options(case, float(np.linalg.norm(b))))
        return dict(kind=kind, S=S, P=P, b=b, x0=np.zeros_like(b))
    if kind == "tetra":
        P = OseenProblem(n_levels=case["levels"], nu=case["nu"], seed=int(seed) % 100000,
                         element="tetra")
        b = P.rhs()
        S = PmSolver(P.descs, **_options(case, float(np.linalg.norm(b))))
        return dict(kind=kind, S=S, b=b, x0=np.zeros_like(b))
    if kind == "batch":
        nus = 10 ** rng.uniform(-2.0, -1.0, case["systems"])
        Ps = [OseenProblem(n_levels=case["levels"], nu=float(nu), seed=int(seed) % 100000 + k)
              for k, nu in enumerate(nus)]
        bs = [P.rhs() for P in Ps]
        norm = min(float(np.linalg.norm(b)) for b in bs)
        S = PmFusedSolver([P.descs for P in Ps], **_options(case, norm))
        return dict(kind=kind, S=S, bs=bs, x0=[np.zeros_like(b) for b in bs])
    assert kind == "step"
    P, D = _channel(*_mesh_key(case))
    L, d = P.n_levels, P.desc(P.n_levels - 1)
    S = PmSolver(D, precision=case["precision"], restart=20, maxit=MAXIT, res_norm_min=1e-300,
                 red_factor=1e-8, red_initial=1)
    n3 = 3 * d.n_udof
    u0 = torch.zeros(n3 + d.n_pdof, dtype=torch.float64, device="cuda")
    u0[:n3] = torch.from_numpy(P.convection_nodal(L - 1)).cuda()
    # another state of the flow for every seed: the perturbed parabola scaled
    # per component
    for c in range(3):
        u0[c * d.n_udof:c * d.n_udof + d.n_active] *= float(rng.uniform(0.8, 1.2))
    return dict(kind=kind, S=S, L=L, n3=n3, u0=u0, u=u0.clone(), w=torch.empty_like(u0),
                f=torch.from_numpy(P.rhs()).cuda() * (case["nu"] * 180.0), nu=case["nu"],
                h=[torch.from_numpy(P.cell_sizes(lev)).cuda() for lev in range(L)],
                conv=[torch.empty(3 * P.desc(lev).n_udof, dtype=torch.float64, device="cuda")
                      for lev in range(L - 1)])


def _ready():
    # the library runs on its own stream: what torch has queued has to be done
    torch.cuda.current_stream().synchronize()


def run(state):
    kind = state["kind"]
    if kind == "mlp":
        loss, grad = state["net"].loss_grad(state["X"], state["T"], want_grad=True)
        return {"loss": loss, "grad": grad}
    S = state["S"]
    if kind == "solve":
        x = state["x"].zero_()
        _ready()
        S.iterate_device(x.data_ptr(), state["b"].data_ptr(), allow=(0, 1))
        return {"u": x[:state["n3"]], "p": x[state["n3"]:]}
    if kind == "vanka":
        return S.cell_vanka(state["level"], state["u"], state["b"], state["sweeps"])
    if kind == "defect":
        return S.coupled_defect(state["level"], state["u"], state["b"])
    if kind == "update":
        S.update_matrices(state["P"].descs)
        return S.iterate(state["x0"], state["b"], allow=(0, 1))[0]
    if kind == "tetra":
        return S.iterate(state["x0"], state["b"], allow=(0, 1))[0]
    if kind == "batch":
        return S.solve(state["x0"], state["bs"], allow=(0, 1))[0]
    tau, theta, L = 1e-3, 0.5, state["L"]
    u, f, w = state["u"].copy_(state["u0"]), state["f"], state["w"]
    _ready()
    conv = state["conv"] + [u]
    for lev in range(L - 1, 0, -1):
        S.interpolate_coarse(lev, conv[lev].data_ptr(), conv[lev - 1].data_ptr())
    for lev in range(L):
        S.assemble_system_level_device(lev, state["h"][lev].data_ptr(), conv[lev].data_ptr(),
                                       state["nu"], 1.0, tau * theta, tau, tau)
    S.refactor()
    S.system_rhs_device(f.data_ptr(), f.data_ptr(), u.data_ptr(), tau * (1 - theta), tau * theta,
                        tau * (1 - theta), w.data_ptr())
    S.iterate_device(u.data_ptr(), w.data_ptr(), allow=(0, 1))
    return u


# -------------------------------------------------------------------- work --
def _hexa_sizes(nx, ny, nz, periodic=False):
    """(active and all nodes, A entries of one block, cells) of a hexahedral mesh."""
    def line(n, per):
        if per:  # all 2n nodes: n vertices couple to 5, n midpoints to 3
            return 2 * n, 8 * n
        return 2 * n - 1, 5 * max(n - 1, 0) + 3 * n
    (ax, ex), (ay, ey), (az, ez) = line(nx, periodic), line(ny, False), line(nz, periodic)
    nodes = (2 * nx + (not periodic)) * (2 * ny + 1) * (2 * nz + (not periodic))
    return ax * ay * az, nodes, ex * ey * ez, nx * ny * nz


def _level_work(act, nodes, nnz, cells, sweeps, defects):
    """Flops of cell-Vanka sweeps (local residuals from the full rows, block
    solve) and defects of one level with one velocity block."""
    per_cell = 2 * (3 * 2197 + 3 * 500 + 3 * 108) + 2 * (3 * 729 + 2 * 324 + 16)
    return sweeps * cells * per_cell + defects * 2 * (3 * nnz + 6 * 108 * cells)


def work(case):
    kind = case["kind"]
    if kind == "mlp":
        rows, weights = case["rows"], 397 * 256 + 256 * 256 + 256 * 85
        return {"bytes": 4 * rows * (397 + 85) + 8 * weights, "flops": 6 * rows * weights}
    if kind in ("tetra", "batch"):
        nx = ny = nz = 2
    else:
        nx, ny, nz = case["nx0"], case["ny0"], case["nz0"]
    L = case["levels"]
    sizes = [_hexa_sizes(nx << k, ny << k, nz << k, kind == "step") for k in range(L)]
    act, nodes, nnz, cells = sizes[-1]
    ndof = 3 * nodes + 4 * cells
    matrix = 12 * nnz + 2 * 28 * 108 * cells + 8 * 3 * nodes  # FP64 values and int32 columns
    if kind == "defect":
        return {"bytes": matrix + 24 * ndof, "flops": _level_work(*sizes[-1], 0, 1)}
    if kind == "vanka":
        return {"bytes": matrix + 24 * ndof + 8 * 1393 * cells,
                "flops": _level_work(*sizes[-1], case["sweeps"], 0)}
    # a solve: the smallest number of iterations that is met in practice
    its = 30 if kind == "step" else 8
    flops = its * (sum(_level_work(*s, 4, 1) for s in sizes[1:]) + _level_work(*sizes[-1], 0, 1)
                   + 4 * its * ndof)
    total = sum(12 * s[2] + 2 * 28 * 108 * s[3] for s in sizes) + 24 * ndof
    if kind == "step":  # assembly and factorisation of every level
        flops += sum(s[3] * (21060 + 6.0e4) for s in sizes)
    if kind == "update":  # nine blocks and the 85x85 LU
        total += sum(64 * s[2] for s in sizes)
        flops += sum(s[3] * 4.1e5 for s in sizes) + its * sum(
            4 * s[3] * 2 * (6 * 2197 + 85 * 85) for s in sizes[1:])
    if kind == "tetra":
        flops, total = 2 * flops, 2 * total
    if kind == "batch":
        flops, total = case["systems"] * flops, case["systems"] * total
    return {"bytes": float(total), "flops": float(flops)}


# ------------------------------------------------------------------- exact --
def _blocks(case, conv, level):
    """FP64 pieces of the Galerkin system of one level, assembled here: per
    cell A [c, 27, 27] and B [3, 4, 27] (the same in every cell)."""
    h, _, ud = _cells(case, level)
    G, phi, dphi, w, pts = _gradients(h)
    n = conv.numel() // 3
    bq = torch.stack([conv[k * n:(k + 1) * n][ud] @ phi.T for k in range(3)], 2)  # [c, q, 3]
    A = case["nu"] * (G[0, 0] + G[1, 1] + G[2, 2]) + torch.zeros(ud.shape[0], 27, 27,
                                                               dtype=torch.float64, device="cuda")
    for s in range(0, ud.shape[0], 4096):
        T = torch.einsum("cqd,qbd->cqb", bq[s:s + 4096], dphi)
        A[s:s + 4096] += torch.einsum("q,qa,cqb->cab", w, phi, T)
    psi = torch.cat([torch.ones_like(pts[:, :1]), pts], 1)
    B = -torch.einsum("q,qm,qbd->dmb", w, psi, dphi)
    return ud, A, B


def _system(case, conv, level):
    """The level's matrix as a sparse CSR tensor with the solver's conventions
    (Dirichlet rows: 1 on the diagonal, no pressure)."""
    P = _mesh(*_mesh_key(case))
    d = P.desc(level)
    nu, na = d.n_udof, d.n_active
    ud, A, B = _blocks(case, conv, level)
    nc = ud.shape[0]
    pd = torch.arange(4 * nc, device="cuda").reshape(nc, 4) + 3 * nu
    rows, cols, vals = [], [], []

    def put(r, c, v):
        keep = v != 0
        rows.append(r[keep])
        cols.append(c[keep])
        vals.append(v[keep])

    act = (ud < na)
    for k in range(3):
        r = (ud + k * nu)[:, :, None].expand(-1, -1, 27)
        put(r, (ud + k * nu)[:, None, :].expand(-1, 27, -1), A * act[:, :, None])
        Bk = B[k].expand(nc, 4, 27)
        r, c = pd[:, :, None].expand(-1, -1, 27), (ud + k * nu)[:, None, :].expand(-1, 4, -1)
        put(r, c, Bk)
        put(c, r, Bk * act[:, None, :])
        i = torch.arange(na, nu, device="cuda") + k * nu
        put(i, i, torch.ones_like(i, dtype=torch.float64))
    n = 3 * nu + 4 * nc
    K = torch.sparse_coo_tensor(torch.stack([torch.cat(rows), torch.cat(cols)]), torch.cat(vals),
                                (n, n)).coalesce()
    return K, ud, pd, nu, na


def _project(r, nu):
    r[3 * nu::4] -= r[3 * nu::4].mean()
    return r


def exact(case, seed):
    kind = case["kind"]
    if kind == "mlp":
        s = prepare(case, seed)
        p = torch.from_numpy(s["net"].params()).double().cuda().requires_grad_()
        x, o = torch.nn.functional.pad(s["X"].double(), (0, 3)), 0
        for n, k in ((256, 400), (256, 256), (96, 256)):  # weights, then biases, layer by layer
            if o:
                x = torch.nn.functional.gelu(x)
            x = x @ p[o:o + n * k].reshape(n, k).T + p[o + n * k:o + n * k + n]
            o += n * k + n
        loss = (x[:, :85] - s["T"].double()).square().mean()
        loss.backward()
        return {"loss": float(loss.detach()), "grad": p.grad.cpu().numpy()}
    if kind == "solve":
        P = _mesh(*_mesh_key(case))
        if P.ndof(-1) > 20000 or P.ndof(-1) < 200:
            return None
        conv, b = _steady(case, seed)
        K, _, _, nu, _ = _system(case, conv[-1], case["levels"] - 1)
        K = K.to_dense()
        b = b.clone()
        K[3 * nu] = 0  # the pressure is given up to a constant
        K[3 * nu, 3 * nu] = 1
        b[3 * nu] = 0
        return {"u": torch.linalg.solve(K, b)[:3 * nu], "p": None}
    if kind not in ("vanka", "defect"):
        return None
    level = case["levels"] - 1
    conv, b = _steady(case, seed)
    u = torch.from_numpy(_state_vector(case, seed)).cuda()
    K, ud, pd, nu, na = _system(case, conv[-1], level)
    K = K.to_sparse_csr()
    if kind == "defect":
        return _project(b - K @ u, nu).cpu().numpy()
    P = _mesh(*_mesh_key(case))
    colour = torch.from_numpy(np.array(P.arrays(level)["cell_colour"])).cuda()
    dofs = torch.cat([ud, ud + nu, ud + 2 * nu, pd], 1)
    crow, col, val = K.crow_indices(), K.col_indices(), K.values()
    n = b.numel()
    keys = torch.repeat_interleave(torch.arange(n, device="cuda"), crow.diff()) * n + col
    for k in range(3):
        u[k * nu + na:(k + 1) * nu] = b[k * nu + na:(k + 1) * nu]
    for _ in range(case["sweeps"]):
        for c in range(int(colour.max()) + 1):
            dd = dofs[colour == c]
            r = (b - K @ u)[dd]
            for s in range(0, dd.shape[0], 1024):
                e = dd[s:s + 1024]
                want = (e[:, :, None] * n + e[:, None, :]).reshape(-1)
                pos = torch.searchsorted(keys, want).clamp_(max=keys.numel() - 1)
                M = torch.where(keys[pos] == want, val[pos], 0.0).reshape(-1, 85, 85)
                u[e] += torch.linalg.solve(M, r[s:s + 1024])
    return u.cpu().numpy()
