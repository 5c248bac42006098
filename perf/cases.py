"""What this framework's speed is measured on: twelve calls a simulation program makes.

The path is: build an edge set's pattern and plans, assemble element maps
into blocked CSR, multiply, solve by CG (plain, mixed precision, with the
learned preconditioner), train that preconditioner, solve many small systems
as one batch.  Sizes are those of this repository's benchmark and tests (the
128^3 and 64^3 tetrahedral lattices, the 10^3 spring box, batches of sheets
of 32..256 vertices a side) and generic ones around them.

Meshes: the five-tet lattice of nx x ny x nz cells; "carved" removes the
tetrahedra inside a ball, so that rows and sizes are uneven; "order" is the
vertex numbering: along a Morton curve with sorted elements, as programs that
reorder their sets have it, or the plain lattice order.
"""
import ctypes
import functools
import math

import numpy as np
import torch

from simit_gb300 import _lib, learned, meshgen, problems
from simit_gb300.runtime import (Context, Mesh, Solver, assemble_heat, assemble_tet_force,
                                 assemble_tet_stiffness, bspmv, call, dtype_code, ptr, solve_opts)

RHO = 1e3
DTYPES = {"f32": torch.float32, "f64": torch.float64}


def listed():
    return [
        # a game-sized spring box: one implicit step, all launches and latency
        {"name": "springs_box_10", "kind": "springs", "nx": 10, "ny": 10, "nz": 10},
        # a new mesh: incidence, pattern, element slots and the assembly plan
        {"name": "mesh_setup_64", "kind": "mesh", "nx": 64, "ny": 64, "nz": 64,
         "order": "morton", "carved": False},
        # the benchmark's assembly: linear elasticity, FP32, element plan
        {"name": "elasticity_assembly_128", "kind": "assembly", "model": "linear", "dtype": "f32",
         "plan": "gather", "nx": 128, "ny": 128, "nz": 128, "order": "morton", "carved": False},
        # a Newton step's tangent and force, FP32, straight from the pattern
        {"name": "neo_newton_64", "kind": "assembly", "model": "neo", "dtype": "f32",
         "plan": "none", "nx": 64, "ny": 64, "nz": 64, "order": "morton", "carved": False},
        # scalar diffusion in FP64, straight from the pattern
        {"name": "heat_assembly_f64_96", "kind": "assembly", "model": "heat", "dtype": "f64",
         "plan": "none", "nx": 96, "ny": 96, "nz": 96, "order": "morton", "carved": False},
        # the FP64 product of a user's own Krylov loop, at the largest size
        {"name": "spmv_f64_128", "kind": "spmv", "bs": 3, "dtype": "f64", "nx": 128, "ny": 128,
         "nz": 128, "order": "morton", "carved": False},
        # the FP32 product on an uneven mesh in the order it was made in
        {"name": "spmv_f32_carved", "kind": "spmv", "bs": 3, "dtype": "f32", "nx": 88, "ny": 61,
         "nz": 97, "order": "lattice", "carved": True},
        # an implicit heat step's solve in FP64, Jacobi CG, one of many right-hand sides
        {"name": "heat_solve_f64_64", "kind": "heat_solve", "nx": 64, "ny": 64, "nz": 64,
         "order": "morton", "carved": False},
        # the headline's step (assembly, refresh, learned PCG) on a smaller mesh
        {"name": "elasticity_step_learned_48", "kind": "step", "precond": "learned", "nx": 48,
         "ny": 48, "nz": 48, "order": "morton", "carved": False},
        # an interactive-sized elasticity step, block Jacobi, uneven mesh
        {"name": "elasticity_step_small", "kind": "step", "precond": "block_jacobi", "nx": 20,
         "ny": 16, "nz": 23, "order": "lattice", "carved": True},
        # one training step of the learned preconditioner: forward, loss, backward, Adam
        {"name": "training_step_32", "kind": "train", "nx": 32, "ny": 32, "nz": 32,
         "order": "lattice", "carved": False},
        # many uneven cloth sheets assembled and solved as one captured graph
        {"name": "cloth_batch_96", "kind": "cloth", "sheets": 96, "lo": 32, "hi": 256},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["springs", "mesh", "assembly", "assembly", "spmv", "spmv", "heat_solve",
                       "step", "train", "cloth"])
    if kind == "cloth":
        hi = _size(rng, 48, 224)
        return {"kind": kind, "sheets": _size(rng, 2, 80), "lo": max(16, hi // 6), "hi": hi}
    top = {"springs": 48, "mesh": 80, "assembly": 100, "spmv": 120, "heat_solve": 64, "step": 44,
           "train": 32}[kind]
    low = {"springs": 4, "mesh": 6, "assembly": 8, "spmv": 6, "heat_solve": 8, "step": 8,
           "train": 10}[kind]
    side = _size(rng, low, top)
    dims = [max(3, int(round(side * math.exp(rng.uniform(-0.25, 0.0))))) for _ in range(3)]
    c = {"kind": kind, "nx": dims[0], "ny": dims[1], "nz": dims[2]}
    if kind == "springs":
        return c
    c["order"] = rng.choice(["morton", "lattice"])
    c["carved"] = bool(rng.random() < 0.4)
    if kind == "assembly":
        c["model"] = rng.choice(["linear", "neo", "heat"])
        c["dtype"] = rng.choice(["f32", "f64"])
        c["plan"] = rng.choice(["gather", "none"])
    elif kind == "spmv":
        c["bs"] = rng.choice([1, 3])
        c["dtype"] = rng.choice(["f32", "f64"])
    elif kind == "step":
        c["precond"] = rng.choice(["learned", "block_jacobi"])
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=1)
def _ctx():
    """The program's one context; its stream is the current one."""
    ctx = Context(0)
    torch.cuda.set_stream(ctx.torch_stream)
    return ctx


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


_EVEN, _ODD = (0, 3, 5, 6), (1, 2, 4, 7)


def _split(corners, center):
    return [center] + [(c, c ^ 1, c ^ 2, c ^ 4) for c in corners]


def _lattice(case):
    """(rest positions [n, 3] float64, tetrahedra [nT, 4] int64) of the case's mesh."""
    d = "cuda"
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    i, j, k = [t.reshape(-1) for t in torch.meshgrid(torch.arange(nx, device=d),
                                                     torch.arange(ny, device=d),
                                                     torch.arange(nz, device=d), indexing="ij")]
    corner = torch.stack([((i + (c & 1)) * (ny + 1) + j + ((c >> 1) & 1)) * (nz + 1) + k + (c >> 2)
                          for c in range(8)], 1)
    par = ((i + j + k) & 1)[:, None, None]
    sel = torch.where(par == 1, torch.tensor(_split(_ODD, _EVEN), device=d)[None],
                      torch.tensor(_split(_EVEN, _ODD), device=d)[None])
    tets = torch.gather(corner[:, None, :].expand(-1, 5, -1), 2, sel).reshape(-1, 4)
    g = torch.stack(torch.meshgrid(torch.arange(nx + 1, device=d), torch.arange(ny + 1, device=d),
                                   torch.arange(nz + 1, device=d), indexing="ij"), -1).reshape(-1, 3)
    if case.get("carved"):
        mid = torch.tensor([nx * 0.4, ny * 0.55, nz * 0.6], device=d)
        away = (g[tets].double().mean(1) - mid).norm(dim=1)
        tets = tets[away > 0.3 * min(nx, ny, nz)]
        used, tets = torch.unique(tets, return_inverse=True)
        g = g[used]
    if case.get("order") == "morton":
        key = torch.zeros(len(g), dtype=torch.int64, device=d)
        for b in range(10):
            for a in range(3):
                key |= ((g[:, a] >> b) & 1) << (3 * b + 2 - a)
        at = torch.argsort(key)
        new = torch.empty_like(at)
        new[at] = torch.arange(len(at), device=d)
        g, tets = g[at], new[tets]
        s = torch.sort(tets, 1).values
        by = torch.argsort(s[:, 2] * len(g) + s[:, 3], stable=True)
        by = by[torch.argsort((s[:, 0] * len(g) + s[:, 1])[by], stable=True)]
        tets = tets[by]
    X = g.double() / torch.tensor([nx, ny, nz], device=d).double()
    e = X[tets[:, :3]] - X[tets[:, 3:]]
    det = (e[:, 0] * torch.linalg.cross(e[:, 1], e[:, 2])).sum(1)
    tets = torch.where((det > 0)[:, None], tets[:, [1, 0, 2, 3]], tets)
    return X, tets


def _shape(X, tets):
    """Inverse shape matrices [nT, 3, 3] and volumes [nT], float64."""
    Ds = (X[tets[:, :3]] - X[tets[:, 3:]]).transpose(1, 2)
    a, b, c = Ds[:, :, 0], Ds[:, :, 1], Ds[:, :, 2]
    rows = torch.stack([torch.linalg.cross(b, c), torch.linalg.cross(c, a),
                        torch.linalg.cross(a, b)], 1)
    det = (a * rows[:, 0]).sum(1)
    return rows / det[:, None, None], -det / 6


def _elastic(case, seed):
    """The elasticity inputs: materials log-uniform over three decades, a
    perturbed state, the bottom face held."""
    X, tets = _lattice(case)
    g = _gen(seed)
    E = 10 ** (3 + 3 * _rand(g, len(tets)))
    nu = 0.35 + 0.1 * _rand(g, len(tets))
    mu = E / (2 * (1 + nu))
    lam = E * nu / ((1 + nu) * (1 - 2 * nu))
    step = 0.02 / max(case["nx"], case["ny"], case["nz"])
    x = X + step * (2 * _rand(g, len(X), 3) - 1)
    v = 0.1 * _randn(g, len(X), 3)
    held = (X[:, 2] == 0).to(torch.int32)
    v[held > 0] = 0
    return {"X": X, "tets": tets, "mu": mu, "lam": lam, "x": x, "v": v, "c": held}


def _assembly_inputs(case, seed):
    s = _elastic(case, seed)
    B, W = _shape(s["X"], s["tets"])
    dt = DTYPES[case["dtype"]]
    out = {"B": B.reshape(-1), "W": W, "x": s["x"].reshape(-1), "v": s["v"].reshape(-1),
           "mu": s["mu"], "lam": s["lam"]}
    if case["model"] == "heat":
        g = _gen(seed + 77)
        out["kappa"] = 10 ** (4 * _rand(g, len(W)) - 2)
        out["T0"] = _rand(g, len(s["X"]))
    out = {k: t.to(dt).contiguous() for k, t in out.items()}
    return dict(out, n=len(s["X"]), tets=s["tets"], c=s["c"])


class _Csr:
    """The assembly pattern of element tuples, from torch alone, with the
    element sum into it."""

    def __init__(self, n, ep):
        self.n, self.card = n, ep.shape[1]
        key = (ep[:, :, None] * n + ep[:, None, :]).reshape(-1)
        uniq, self.slot = torch.unique(key, return_inverse=True)
        self.rows, self.cols = uniq // n, uniq % n
        self.nnzb = len(uniq)
        self.slot = self.slot.reshape(len(ep), -1)
        count = torch.bincount(self.rows, minlength=n)
        self.rowptr = torch.cat([count.new_zeros(1), count.cumsum(0)]).to(torch.int32)
        self.colidx = self.cols.to(torch.int32)

    def add(self, vals, i, j, block):
        vals.index_add_(0, self.slot[:, i * self.card + j], block)

    def scalar(self, vals, bs):
        """The matrix as a torch CSR tensor of scalars."""
        r = self.rows[:, None, None] * bs + torch.arange(bs, device="cuda")[None, :, None]
        c = self.cols[:, None, None] * bs + torch.arange(bs, device="cuda")[None, None, :]
        shape = (self.nnzb, bs, bs)
        r, c = r.expand(shape).reshape(-1), c.expand(shape).reshape(-1)
        at = torch.argsort(r, stable=True)
        ptr_ = torch.cat([r.new_zeros(1), torch.bincount(r, minlength=self.n * bs).cumsum(0)])
        return torch.sparse_csr_tensor(ptr_.to(torch.int32), c[at].to(torch.int32),
                                       vals.reshape(-1).double()[at],
                                       size=(self.n * bs, self.n * bs))


def _grads(B):
    return torch.cat([B, -B.sum(1, keepdim=True)], 1)


def _tet_matrix(model, p, B, x, tets, c, W, mu, lam, h):
    """Stiffness h^2 K plus lumped mass in float64: the linear model's, or the
    neo-Hookean tangent with q = F^-T g in the place of g where it belongs."""
    g = _grads(B)
    free = (c <= 0)[tets].double()
    q, cc = g, mu
    if model == "neo":
        F = (x[tets[:, :3]] - x[tets[:, 3:]]).transpose(1, 2) @ B
        q = g @ torch.linalg.inv(F)
        cc = mu - lam * torch.log(torch.linalg.det(F))
    vals = torch.zeros(p.nnzb, 3, 3, dtype=torch.float64, device="cuda")
    eye = torch.eye(3, dtype=torch.float64, device="cuda")
    for i in range(4):
        for j in range(4):
            qi, qj = q[:, i], q[:, j]
            k = lam[:, None, None] * qi[:, :, None] * qj[:, None, :]
            k += cc[:, None, None] * qj[:, :, None] * qi[:, None, :]
            k += (mu * (g[:, i] * g[:, j]).sum(1))[:, None, None] * eye
            k *= (h * h * W * free[:, i] * free[:, j])[:, None, None]
            if i == j:
                k += (0.25 * RHO * W)[:, None, None] * eye
            p.add(vals, i, j, k)
    return vals


def _tet_force(model, n, B, x, v, tets, c, W, mu, lam, h, grav):
    F = (x[tets[:, :3]] - x[tets[:, 3:]]).transpose(1, 2) @ B
    eye = torch.eye(3, dtype=torch.float64, device="cuda")
    if model == "neo":
        Fi = torch.linalg.inv(F).transpose(1, 2)
        P = mu[:, None, None] * (F - Fi) + (lam * torch.log(torch.linalg.det(F)))[:, None, None] * Fi
    else:
        D = F - eye
        P = mu[:, None, None] * (D + D.transpose(1, 2))
        P += (lam * D.diagonal(dim1=1, dim2=2).sum(1))[:, None, None] * eye
    H = -W[:, None, None] * (P @ B.transpose(1, 2))
    H = torch.cat([H, -H.sum(2, keepdim=True)], 2)
    m = 0.25 * RHO * W
    f = torch.zeros(n, 3, dtype=torch.float64, device="cuda")
    for i in range(4):
        fi = h * H[:, :, i] + m[:, None] * (h * grav + v[tets[:, i]])
        f.index_add_(0, tets[:, i], fi * (c <= 0)[tets[:, i]].double()[:, None])
    return f


def _heat_matrix(p, B, W, kappa, dt, T0, tets):
    g = _grads(B)
    vals = torch.zeros(p.nnzb, dtype=torch.float64, device="cuda")
    b = torch.zeros(p.n, dtype=torch.float64, device="cuda")
    for i in range(4):
        for j in range(4):
            m = W / 20 * (2 if i == j else 1)
            p.add(vals, i, j, m + dt * kappa * W * (g[:, i] * g[:, j]).sum(1))
            b.index_add_(0, tets[:, i], m * T0[tets[:, j]])
    return vals, b


GRAV = (0.0, 0.0, -9.81)
NEO_H, HEAT_DT, SOLVE_DT = 0.01, 1e-2, 1e-3


def _stiff(case, seed):
    """The elasticity system in float64 (h = 1, linear): pattern, values, force."""
    s = _elastic(case, seed)
    p = _Csr(len(s["X"]), s["tets"])
    B, W = _shape(s["X"], s["tets"])
    A = _tet_matrix("linear", p, B, s["x"], s["tets"], s["c"], W, s["mu"], s["lam"], 1.0)
    return s, p, A, B, W


def _springs_inputs(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    L = meshgen.springs_lattice(nx, ny, nz, 0.1, 0.01, seed)
    g = meshgen.rng(seed + 5)
    n = L["n"]
    v = 0.1 * g.normal(size=(n, 3))
    v[L["fixed"] > 0] = 0
    return dict(L, v=v.reshape(-1), m=np.ones(n), k=10 ** g.uniform(3.5, 4.5, len(L["l0"])),
                h=1e-3)


@functools.lru_cache(maxsize=512)
def _sheet(side):
    return meshgen.cloth_sheet(side)


def _cloth_inputs(case, seed):
    c = problems.CLOTH
    sides = problems.cloth_sides(case["sheets"], case["lo"], case["hi"])
    g = meshgen.rng(seed)
    parts, off = [], 0
    for s in sides:
        sh = _sheet(int(s))
        x = sh["x"].reshape(-1, 3).copy()
        x[:, 2] += g.uniform(-0.2, 0.2, len(x)) / (s - 1)
        parts.append((x.reshape(-1), sh["ep"] + off,
                      np.where(sh["is_bend"] > 0, c["k_bend"], c["k_stretch"]), sh["l0"],
                      sh["fixed"]))
        off += sh["n"]
    x, ep, k, l0, fixed = [np.concatenate(t) for t in zip(*parts)]
    ends = np.concatenate([[0], np.cumsum(np.asarray(sides, np.int64) ** 2)]).astype(np.int32)
    return {"n": off, "x": x, "ep": ep.astype(np.int32), "k": k, "l0": l0, "fixed": fixed,
            "sys_ptr": ends, "sides": np.asarray(sides)}


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------
def prepare(case, seed):
    ctx = _ctx()
    kind = case["kind"]
    st = {"kind": kind, "ctx": ctx}
    if kind == "springs":
        L = _springs_inputs(case, seed)
        mesh = Mesh(ctx, L["n"], L["ep"], 2)
        t = {k: torch.tensor(L[k], device="cuda") for k in ("x", "v", "m", "fixed", "k", "l0")}
        vals = mesh.empty(mesh.nnzb * 9, torch.float64)
        f = mesh.empty(mesh.n * 3, torch.float64)
        vals.view(-1, 9)[:, ::4] = 1.0
        S = Solver(ctx, mesh.n, 3, mesh.pattern.rowptr, mesh.pattern.colidx, vals, mesh.nnzb,
                   solve_opts(precision=_lib.SOLVE_F64, precond=_lib.PRECOND_NONE, tol=1e-8,
                              maxiters=10000))
        st.update(t, mesh=mesh, vals=vals, f=f, S=S, h=L["h"])
    elif kind == "mesh":
        X, tets = _lattice(case)
        g = _gen(seed)  # another numbering inside each element: other slots, same mesh
        by = torch.argsort(_rand(g, len(tets), 4), 1)
        st.update(n=len(X), ep=torch.gather(tets, 1, by).to(torch.int32).reshape(-1).contiguous())
    elif kind == "assembly":
        a = _assembly_inputs(case, seed)
        a["mesh"] = Mesh(ctx, a["n"], a["tets"].to(torch.int32).reshape(-1), 4,
                         plan=None if case["plan"] == "none" else case["plan"])
        del a["tets"]
        st.update(a, model=case["model"], dt=DTYPES[case["dtype"]])
    elif kind == "spmv":
        s, p, A, B, W = _stiff(case, seed)
        if case["bs"] == 1:
            g = _gen(seed + 77)
            A, _ = _heat_matrix(p, B, W, 10 ** (4 * _rand(g, len(W)) - 2), HEAT_DT, s["X"][:, 0],
                                s["tets"])
        dt = DTYPES[case["dtype"]]
        st.update(n=p.n, bs=case["bs"], rowptr=p.rowptr, colidx=p.colidx,
                  vals=A.reshape(-1).to(dt), x=_randn(_gen(seed + 1), p.n * case["bs"]).to(dt))
        st["y"] = torch.empty_like(st["x"])
    elif kind == "heat_solve":
        a = _heat_system(case, seed)
        p = a["p"]
        S = Solver(ctx, p.n, 1, p.rowptr, p.colidx, a["A"], p.nnzb,
                   solve_opts(precision=_lib.SOLVE_F64, precond=_lib.PRECOND_JACOBI, tol=1e-11,
                              maxiters=100000))
        st.update(S=S, b=a["b"], x=torch.zeros_like(a["b"]))
    elif kind == "step":
        s = _elastic(case, seed)
        host = {"n": len(s["X"]), "tets": s["tets"].to(torch.int32).reshape(-1).cpu().numpy(),
                "X0": s["X"].reshape(-1).cpu().numpy(), "x": s["x"].reshape(-1).cpu().numpy(),
                "mu": s["mu"].cpu().numpy(), "lam": s["lam"].cpu().numpy(),
                "c": s["c"].cpu().numpy()}
        prm, pc = None, _lib.PRECOND_BLOCK_JACOBI
        if case["precond"] == "learned":
            prm, pc = torch.tensor(learned.load_weights("sym"), device="cuda"), _lib.PRECOND_LEARNED
        st["p"] = problems.HeteroElasticity(ctx, host, dtype=torch.float32, precond=pc,
                                            learned_params=prm)
    elif kind == "train":
        s, p, A, _, _ = _stiff(case, seed)
        A = A.reshape(-1).float()
        mesh = _PatternOf(p)
        r, e, eAe = _train_pair(case, seed, s, p, A)
        tr = learned.Trainer(ctx, params=learned.load_weights("sym"), lr=5e-5)
        st.update(mesh=mesh, A=A, graph=learned.Graph(ctx, mesh, A, form="sym"), tr=tr, r=r, e=e,
                  eAe=eAe)
    else:
        st["cb"] = problems.ClothBatch(ctx, _cloth_inputs(case, seed))
        st["cb"].capture()
    return st


class _PatternOf:
    """A mesh's pattern as learned.Graph reads it."""

    def __init__(self, p):
        self.n, self.nnzb, self.pattern = p.n, p.nnzb, self
        self.rowptr, self.colidx = p.rowptr, p.colidx


def _train_pair(case, seed, s, p, A):
    """A smooth-plus-rough correction e and its residual r = A e."""
    g = _gen(seed + 3)
    w = 2 * math.pi * (1 + 3 * _rand(g, 4, 3))
    e = sum(torch.sin(s["X"] @ w[q] + q)[:, None] * _randn(g, 1, 3) for q in range(4))
    e = (e + 0.05 * _randn(g, p.n, 3)) * (s["c"] <= 0).double()[:, None]
    e = e.float().reshape(-1)
    r = p.scalar(A, 3) @ e.double()
    return r.float(), e, float(e.double() @ r)


def _heat_system(case, seed):
    X, tets = _lattice(case)
    g = _gen(seed + 77)
    B, W = _shape(X, tets)
    p = _Csr(len(X), tets)
    A, b = _heat_matrix(p, B, W, 10 ** (4 * _rand(g, len(W)) - 2), SOLVE_DT, _rand(g, len(X)),
                        tets)
    return {"p": p, "A": A, "b": b}


def run(st):
    kind, ctx = st["kind"], st["ctx"]
    if kind == "springs":
        m = st["mesh"]
        call("sg_assemble_springs", ctx.h, m.ref(), _lib.F64, 0, ptr(st["x"]), ptr(st["v"]),
             ptr(st["m"]), ptr(st["fixed"]), ptr(st["k"]), ptr(st["l0"]), st["h"], 0.0,
             (ctypes.c_double * 3)(*GRAV), ptr(st["vals"]), ptr(st["f"]), 1)
        st["S"].refresh()
        v = st["v"].clone()
        st["S"].solve(st["f"], v)
        return {"matrix": st["vals"], "force": st["f"], "v": v, "x": st["x"] + st["h"] * v}
    if kind == "mesh":
        m = Mesh(ctx, st["n"], st["ep"], 4, plan="gather")
        p = m.pattern
        return {"ve_ptr": p.ve_ptr, "ve_idx": p.ve_idx, "rowptr": p.rowptr, "colidx": p.colidx,
                "slots": p.slots, "slot_src_ptr": m.slot_src_ptr, "slot_src": m.slot_src}
    if kind == "assembly":
        m, dt = st["mesh"], st["dt"]
        if st["model"] == "heat":
            A, b = assemble_heat(m, st["B"], st["W"], st["kappa"], HEAT_DT, st["T0"], dtype=dt,
                                 exact=False)
            return {"matrix": A, "rhs": b}
        mod, h = {"linear": (_lib.MODEL_LINEAR, 1.0),
                  "neo": (_lib.MODEL_NEOHOOKEAN, NEO_H)}[st["model"]]
        A = assemble_tet_stiffness(m, mod, st["x"], st["c"], st["B"], st["W"], st["mu"], st["lam"],
                                   h, RHO, dtype=dt, exact=False)
        f = assemble_tet_force(m, mod, st["x"], st["v"], st["c"], st["B"], st["W"], st["mu"],
                               st["lam"], h, RHO, np.array(GRAV), dtype=dt, exact=False)
        return {"matrix": A, "force": f}
    if kind == "spmv":
        return bspmv(ctx, st["n"], st["bs"], st["rowptr"], st["colidx"], st["vals"], st["x"],
                     st["y"])
    if kind == "heat_solve":
        st["S"].solve_ex(st["b"], st["x"], x_zero=True)
        return st["x"]
    if kind == "step":
        # the FP32 simulation keeps its displacements in FP32
        p = st["p"]
        p.step()
        return {"matrix": p.A, "force": p.f, "displacement": p.u.float()}
    if kind == "train":
        tr = st["tr"]
        loss = tr.step(st["graph"], st["r"], st["e"], st["eAe"])
        return {"loss": loss, "grad": tr.grad, "params": tr.params, "m": tr.m, "v": tr.v}
    st["cb"].replay()
    return {"matrix": st["cb"].A, "force": st["cb"].f, "v": st["cb"].vout}


def _counts(case):
    """(vertices, elements, pattern entries) of the case, carving left out."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = (nx + 1) * (ny + 1) * (nz + 1)
    cells = nx * ny * nz
    axis = nx * (ny + 1) * (nz + 1) + (nx + 1) * ny * (nz + 1) + (nx + 1) * (ny + 1) * nz
    face = nx * ny * (nz + 1) + nx * (ny + 1) * nz + (nx + 1) * ny * nz
    nE, nnzb = 5 * cells, n + 2 * (axis + face)
    if case.get("carved"):
        keep = 1 - 4.0 / 3 * math.pi * (0.3 * min(nx, ny, nz)) ** 3 / cells
        n, nE, nnzb = int(n * keep), int(nE * keep), int(nnzb * keep)
    return n, nE, nnzb


def work(case):
    kind = case["kind"]
    if kind == "cloth":
        sides = problems.cloth_sides(case["sheets"], case["lo"], case["hi"]).astype(np.int64)
        n = int((sides ** 2).sum())
        nE, nnzb = 6 * n, 13 * n
        return {"bytes": nE * 16 + n * 42 + nnzb * 40 + n * 24, "flops": nE * 60 + nnzb * 18}
    if kind == "springs":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        n = nx * ny * nz
        nE = (nx - 1) * ny * nz + nx * (ny - 1) * nz + nx * ny * (nz - 1)
        nnzb = n + 2 * nE
        return {"bytes": nE * 24 + n * 57 + nnzb * 76 + n * 72, "flops": nE * 60 + nnzb * 18}
    n, nE, nnzb = _counts(case)
    if kind == "mesh":
        return {"bytes": nE * (16 + 16 + 64 + 64) + n * 8 + nnzb * 8, "flops": 0}
    if kind == "assembly":
        s = 4 if case["dtype"] == "f32" else 8
        if case["model"] == "heat":
            return {"bytes": nE * (16 + 11 * s) + n * 2 * s + nnzb * s, "flops": nE * 150}
        return {"bytes": nE * (16 + 12 * s) + n * (4 + 9 * s) + nnzb * 9 * s, "flops": nE * 1200}
    if kind == "spmv":
        s, bs = 4 if case["dtype"] == "f32" else 8, case["bs"]
        return {"bytes": nnzb * (4 + s * bs * bs) + n * (4 + 2 * s * bs),
                "flops": 2 * nnzb * bs * bs}
    if kind == "heat_solve":
        return {"bytes": nnzb * 12 + n * 20, "flops": 2 * nnzb}
    if kind == "step":
        return {"bytes": nE * 64 + n * 28 + nnzb * 40 + n * 36, "flops": nE * 1200 + 18 * nnzb}
    H, K = learned.H, learned.K  # forward, its transpose, and two backward passes of each
    net = n * 2 * (2 * H * H + 4 * K * H + 9 * H) + nnzb * 2 * (3 + 2 * K)
    return {"bytes": nnzb * 40 + n * 24 + learned.nparams() * 20, "flops": 6 * net}


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------
def _cg(A, b, x, dinv, tol, maxiters):
    r = b - A @ x
    z = dinv * r
    p, rz, stop = z.clone(), r @ z, tol * tol * (b @ b)
    for it in range(maxiters):
        q = A @ p
        a = rz / (p @ q)
        x = x + a * p
        r = r - a * q
        if it % 25 == 24 and float(r @ r) <= float(stop):
            break
        z = dinv * r
        new = r @ z
        p = z + (new / rz) * p
        rz = new
    return x


def _diag(p, vals, bs):
    d = torch.empty(p.n, bs, dtype=torch.float64, device="cuda")
    on = p.rows == p.cols
    d[p.rows[on]] = vals.reshape(-1, bs, bs)[on].diagonal(dim1=1, dim2=2).double()
    return d.reshape(-1)


def _spring_system(n, x, v, m, fixed, ep, k, l0, h):
    """The springs' system in float64: pattern, blocks, force."""
    p = _Csr(n, ep)
    d = x[ep[:, 1]] - x[ep[:, 0]]
    L = d.norm(dim=1)
    U = d / L[:, None]
    f0 = k * (L - l0)
    eye = torch.eye(3, dtype=torch.float64, device="cuda")
    kb = (k - f0 / L)[:, None, None] * U[:, :, None] * U[:, None, :]
    kb = h * h * (kb + (f0 / L)[:, None, None] * eye)
    free = (fixed == 0).double()
    fe = (h * f0)[:, None] * U
    vals = torch.zeros(p.nnzb, 3, 3, dtype=torch.float64, device="cuda")
    f = torch.zeros(n, 3, dtype=torch.float64, device="cuda")
    for i in range(2):
        fi = free[ep[:, i]]
        for j in range(2):
            w = fi * free[ep[:, j]] if i != j else fi
            p.add(vals, i, j, (w if i == j else -w)[:, None, None] * kb)
        f.index_add_(0, ep[:, i], (fi if i == 0 else -fi)[:, None] * fe)
    on = p.rows == p.cols
    held = torch.zeros(3, 3, dtype=torch.float64, device="cuda")
    held[0, 0] = 1
    md = free[:, None, None] * m[:, None, None] * eye + (1 - free)[:, None, None] * held
    vals[on] += md[p.rows[on]]
    grav = torch.tensor(GRAV, dtype=torch.float64, device="cuda")
    f += free[:, None] * (m[:, None] * v + (h * m)[:, None] * grav)
    return p, vals, f


def _solve_springs(p, vals, f, x0, tol):
    """The blocks' solution; a held point's empty rows keep their start value."""
    d = _diag(p, vals, 3)
    return _cg(p.scalar(vals, 3), f.reshape(-1), x0.reshape(-1),
               torch.where(d == 0, torch.ones_like(d), 1 / d), tol, 3000)


def exact(case, seed):
    _ctx()
    kind = case["kind"]
    if kind == "mesh":
        return None
    if kind == "springs":
        L = _springs_inputs(case, seed)
        t = {k: torch.tensor(L[k], device="cuda") for k in ("x", "v", "m", "fixed", "k", "l0")}
        ep = torch.tensor(L["ep"], device="cuda").long().reshape(-1, 2)
        x, v = t["x"].reshape(-1, 3), t["v"].reshape(-1, 3)
        p, A, f = _spring_system(L["n"], x, v, t["m"], t["fixed"], ep, t["k"], t["l0"], L["h"])
        u = _solve_springs(p, A, f, v, 1e-15)
        return {"matrix": A.reshape(-1), "force": f.reshape(-1), "v": u,
                "x": t["x"] + L["h"] * u}
    if kind == "assembly":
        a = {k: t.double() if torch.is_tensor(t) and t.is_floating_point() else t
             for k, t in _assembly_inputs(case, seed).items()}
        p = _Csr(a["n"], a["tets"])
        B, x, v = a["B"].reshape(-1, 3, 3), a["x"].reshape(-1, 3), a["v"].reshape(-1, 3)
        if case["model"] == "heat":
            A, b = _heat_matrix(p, B, a["W"], a["kappa"], HEAT_DT, a["T0"], a["tets"])
            return {"matrix": A, "rhs": b}
        h = NEO_H if case["model"] == "neo" else 1.0
        rest = (a["tets"], a["c"], a["W"], a["mu"], a["lam"], h)
        grav = torch.tensor(GRAV, dtype=torch.float64, device="cuda")
        A = _tet_matrix(case["model"], p, B, x, *rest)
        f = _tet_force(case["model"], p.n, B, x, v, *rest, grav)
        return {"matrix": A.reshape(-1), "force": f.reshape(-1)}
    if kind == "spmv":
        st = prepare(case, seed)
        n, bs = st["n"], st["bs"]
        per = (st["rowptr"][1:] - st["rowptr"][:-1]).long()
        rows = torch.repeat_interleave(torch.arange(n, device="cuda"), per)
        A, x = st["vals"].reshape(-1, bs, bs), st["x"].double().reshape(n, bs)
        y = torch.zeros(n, bs, dtype=torch.float64, device="cuda")
        for at in range(0, len(rows), 1 << 23):
            s = slice(at, at + (1 << 23))
            y.index_add_(0, rows[s], (A[s].double() * x[st["colidx"][s].long()][:, None, :]).sum(2))
        return y.reshape(-1)
    if kind == "heat_solve":
        a = _heat_system(case, seed)
        return _cg(a["p"].scalar(a["A"], 1), a["b"], torch.zeros_like(a["b"]),
                   1 / _diag(a["p"], a["A"], 1), 1e-15, 3000)
    if kind == "step":
        s, p, A, B, W = _stiff(case, seed)
        grav = torch.tensor(GRAV, dtype=torch.float64, device="cuda")
        f = _tet_force("linear", p.n, B, s["x"], torch.zeros_like(s["x"]), s["tets"], s["c"], W,
                       s["mu"], s["lam"], 1.0, grav).reshape(-1)
        u = _cg(p.scalar(A, 3), f, torch.zeros_like(f), 1 / _diag(p, A, 3), 1e-12, 8000)
        return {"matrix": A.reshape(-1), "force": f, "displacement": u}
    if kind == "train":
        return _exact_training(case, seed)
    h = _cloth_inputs(case, seed)
    c = problems.CLOTH
    d = {k: torch.tensor(h[k], device="cuda") for k in ("x", "fixed", "k", "l0")}
    x = d["x"].float().double().reshape(-1, 3)
    p, A, f = _spring_system(h["n"], x, torch.zeros_like(x),
                             torch.full((h["n"],), c["mass"], device="cuda").double(), d["fixed"],
                             torch.tensor(h["ep"], device="cuda").long().reshape(-1, 2),
                             d["k"].float().double(), d["l0"].float().double(), c["dt"])
    v = _solve_springs(p, A, f, torch.zeros_like(f), 1e-13)
    return {"matrix": A.reshape(-1), "force": f.reshape(-1), "v": v}


def _exact_training(case, seed):
    """One training step of the symmetric network in float64, by autograd:
    M = L^-T (I + N)^T (I + N) L^-1 with the linear three-layer network N and
    bfloat16 64x64 weights."""
    s, p, A, _, _ = _stiff(case, seed)
    A = A.reshape(-1).float().double()
    r, e, eAe = _train_pair(case, seed, s, p, A.float())
    r, e, n = r.double().reshape(-1, 3), e.double().reshape(-1, 3), p.n
    blocks = A.reshape(-1, 3, 3)
    on = p.rows == p.cols
    D = torch.empty(n, 3, 3, dtype=torch.float64, device="cuda")
    D[p.rows[on]] = blocks[on]
    Li = torch.linalg.inv(torch.linalg.cholesky(D))
    norm = blocks.flatten(1).norm(dim=1)
    dn = torch.empty(n, dtype=torch.float64, device="cuda")
    dn[p.rows[on]] = norm[on]
    w = norm / torch.sqrt(dn[p.rows] * dn[p.cols])
    w = torch.where(on, torch.zeros_like(w), w)
    G = torch.sparse_csr_tensor(p.rowptr, p.colidx, w, size=(n, n))

    class Agg(torch.autograd.Function):  # G is symmetric
        @staticmethod
        def forward(ctx, t):
            return G @ t

        @staticmethod
        def backward(ctx, t):
            return G @ t.contiguous()

    flat = torch.tensor(learned.load_weights("sym"), device="cuda").double()
    W, at = {}, 0
    for name, (a, b) in learned.SHAPES:
        W[name] = flat[at:at + a * b].reshape(a, b).clone().requires_grad_()
        at += a * b
    half = {k: W[k] + (W[k].detach().float().bfloat16().double() - W[k].detach())
            for k in ("W2h", "W3h")}

    def net(x):  # N x
        h1 = x @ W["W1s"].T + Agg.apply(x) @ W["W1m"].T
        h2 = h1 @ half["W2h"].T + Agg.apply(h1 @ W["P2"].T) @ W["W2m"].T
        h3 = h2 @ half["W3h"].T + Agg.apply(h2 @ W["P3"].T) @ W["W3m"].T
        return h3 @ W["Wout"].T

    def net_t(y):  # N^T y
        h3 = y @ W["Wout"]
        h2 = h3 @ half["W3h"] + Agg.apply(h3 @ W["W3m"]) @ W["P3"]
        h1 = h2 @ half["W2h"] + Agg.apply(h2 @ W["W2m"]) @ W["P2"]
        return h1 @ W["W1s"] + Agg.apply(h1 @ W["W1m"])

    x = (Li @ r[:, :, None])[:, :, 0]
    y = x + net(x)
    z = (Li.transpose(1, 2) @ (y + net_t(y))[:, :, None])[:, :, 0]
    K = p.scalar(A, 3)
    diff = (z - e).reshape(-1)
    Ad = K @ diff.detach()
    loss = float(diff.detach() @ Ad) / eAe
    z.backward((2 / eAe * Ad).reshape(-1, 3))
    grad = torch.cat([W[name].grad.reshape(-1) for name, _ in learned.SHAPES])
    m, v = 0.1 * grad, 0.001 * grad * grad
    params = flat - 5e-5 * (m / 0.1) / ((v / 0.001).sqrt() + 1e-8)
    return {"loss": loss, "grad": grad, "params": params, "m": m, "v": v}
