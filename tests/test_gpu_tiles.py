"""GPU checks of the row-tile assembly at the sizes where it changes path:
rows longer than a tile can address, rows of more than one mask word, meshes
whose numbering shares few elements between neighbouring rows (a tile taken
in parts), elements that list a vertex twice, vertices without elements, and
meshes of fewer rows than a tile.  Exact mode against the oracle bit for
bit; the contracted kernels within 1e-12 of the largest value in FP64 and
1e-5 in FP32 (about 300 terms a sum at most, each rounded a few times)."""
import numpy as np
import pytest
import torch

from simit_gb300 import _lib, meshgen

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(gpu_ctx):
    return gpu_ctx


def _np(t):
    return t.detach().cpu().numpy()


def _springs(kind):
    """(n, endpoints): hub = vertex 0 in 400 springs (a row past 8-bit
    positions) and vertex 1 in 90 (three mask words); random = every second
    vertex unused; tiny = one spring."""
    g = meshgen.rng(21)
    if kind == "tiny":
        return 2, np.array([[1, 0]])
    if kind == "random":
        return 700, 2 * g.integers(0, 350, size=(2500, 2))
    hub = np.stack([np.zeros(400, int), 2 + np.arange(400)], 1)
    two = np.stack([2 + g.permutation(400)[:90], np.ones(90, int)], 1)
    ep = np.concatenate([hub, two, g.integers(2, 402, size=(300, 2))])
    return 402, ep[g.permutation(len(ep))]


@pytest.mark.parametrize("kind", ["tiny", "random", "hub"])
@pytest.mark.parametrize("form", [0, 1])
def test_springs(ctx, oracle, kind, form):
    from simit_gb300.runtime import Mesh, assemble_springs
    n, ep = _springs(kind)
    ep = ep[ep[:, 0] != ep[:, 1]]
    # the oracle wants every vertex in some element (a diagonal block each)
    used, ep = np.unique(ep, return_inverse=True)
    n, ep = len(used), ep.reshape(-1, 2)
    g = meshgen.rng(5)
    x, v = g.normal(size=n * 3), g.normal(size=n * 3)
    m, k = g.uniform(1, 2, n), g.uniform(10, 20, len(ep))
    l0 = g.uniform(0.5, 1, len(ep))
    fixed = (g.uniform(size=n) < 0.2).astype(np.uint8)
    grav = np.array([0.1, 0.2, -9.81])
    mesh = Mesh(ctx, n, ep.astype(np.int32).reshape(-1), 2)
    rp, ci = mesh.pattern.host()
    oA, of = oracle.springs_assemble(form, x, v, m, fixed, mesh.pattern.endpoints.cpu().numpy(),
                                     k, l0, 0.01, 0.1, grav, rp, ci)
    A, f = assemble_springs(mesh, x, v, m, fixed, k, l0, 0.01, 0.1, grav, form=form)
    ctx.sync()
    assert np.array_equal(_np(A), oA) and np.array_equal(_np(f), of)
    A, f = assemble_springs(mesh, x, v, m, fixed, k, l0, 0.01, 0.1, grav, form=form,
                            dtype=torch.float32, exact=False)
    ctx.sync()
    assert np.abs(_np(A) - oA).max() <= 1e-5 * np.abs(oA).max()
    assert np.abs(_np(f) - of).max() <= 1e-5 * np.abs(of).max()


@pytest.mark.parametrize("kind", ["tiny", "random", "hub"])
def test_repeated_endpoints(ctx, kind):
    """Scalar springs, some of them from a vertex to itself, against the
    same blocks through the row owners, bit for bit."""
    from simit_gb300.runtime import Mesh, assemble_blocks, assemble_scalar_springs
    n, ep = _springs(kind)
    ep = ep.copy()
    ep[::5, 1] = ep[::5, 0]
    a = meshgen.rng(6).normal(size=len(ep))
    eb = np.stack([a, -a, -a, a], 1)
    mesh = Mesh(ctx, n, ep.astype(np.int32).reshape(-1), 2)
    ref = assemble_blocks(mesh, eb, 1, exact=True)
    got = assemble_scalar_springs(mesh, a, 0.0, 1.0)
    ctx.sync()
    assert torch.equal(got, ref)


def _tets(kind):
    """(positions [n, 3], tets): lattice, its vertices renumbered at random
    (with elements in random order too), or a fan of tetrahedra around one
    edge (two vertices in 130 elements, rows of 132 blocks)."""
    g = meshgen.rng(8)
    if kind == "fan":
        t = np.linspace(0, 2 * np.pi, 131)[:-1]
        ring = np.stack([np.cos(t), np.sin(t), 0.1 * np.sin(7 * t)], 1)
        X = np.concatenate([[[0, 0, -1.0], [0, 0, 1.0]], ring])
        k = np.arange(130)
        T = np.stack([np.zeros(130, int), np.ones(130, int), 2 + k, 2 + (k + 1) % 130], 1)
    else:
        mg = meshgen.tet_grid(9, 8, 7)
        X, T = mg["X0"].reshape(-1, 3), mg["tets"].reshape(-1, 4).astype(int)
        if kind == "random":
            new = g.permutation(len(X))
            Y = np.empty_like(X)
            Y[new] = X
            X, T = Y, new[T][g.permutation(len(T))]
    d = X[T[:, :3]] - X[T[:, 3:]]
    flip = np.einsum("ti,ti->t", d[:, 0], np.cross(d[:, 1], d[:, 2])) > 0
    T[flip, 0], T[flip, 1] = T[flip, 1].copy(), T[flip, 0].copy()
    return X, T


@pytest.mark.parametrize("kind", ["lattice", "random", "fan"])
@pytest.mark.parametrize("plan", [None, "gather"])
def test_tets(ctx, oracle, kind, plan):
    from simit_gb300.runtime import (Mesh, assemble_heat, assemble_tet_force,
                                     assemble_tet_stiffness, tet_precompute)
    X, T = _tets(kind)
    n, nT = len(X), len(T)
    tets = T.astype(np.int32).reshape(-1)
    g = meshgen.rng(9)
    x = X.reshape(-1) + g.uniform(-1e-3, 1e-3, n * 3)
    v = g.normal(size=n * 3)
    mu, lam = g.uniform(1e3, 1e5, nT), g.uniform(1e3, 1e5, nT)
    c = (g.uniform(size=n) < 0.2).astype(np.int32)
    kappa, T0 = 10 ** g.uniform(-2, 2, nT), g.uniform(size=n)
    grav = np.array([0.1, 0.2, -9.81])
    mesh = Mesh(ctx, n, tets, 4, plan=plan)
    rp, ci = mesh.pattern.host()
    oB, oW, _ = oracle.tet_precompute(X.reshape(-1), tets, 1e3)
    B, W, _ = tet_precompute(mesh, X.reshape(-1), 1e3)
    oA, ob = oracle.heat_assemble(n, tets, oB, oW, kappa, 1e-2, T0, rp, ci)
    A, b = assemble_heat(mesh, B, W, kappa, 1e-2, T0)
    ctx.sync()
    assert np.array_equal(_np(A), oA) and np.array_equal(_np(b), ob)

    def close(got, ref, tol):
        ctx.sync()
        assert np.abs(_np(got) - ref).max() <= tol * np.abs(ref).max()

    for dt, tol in ((torch.float64, 1e-12), (torch.float32, 1e-5)):
        A, b = assemble_heat(mesh, B, W, kappa, 1e-2, T0, dtype=dt, exact=False)
        close(A, oA, tol)
        close(b, ob, tol)
    for model in (0, 1):
        oK = oracle.tet_stiffness(model, x, c, tets, oB, oW, mu, lam, 0.01, 1e3, rp, ci)
        of = oracle.tet_force(model, x, v, c, tets, oB, oW, mu, lam, 0.01, 1e3, grav)
        K = assemble_tet_stiffness(mesh, model, x, c, B, W, mu, lam, 0.01, 1e3, exact=False)
        f = assemble_tet_force(mesh, model, x, v, c, B, W, mu, lam, 0.01, 1e3, grav, exact=False)
        close(K, oK, 1e-12)
        close(f, of, 1e-12)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("exact", [False, True])
def test_heat_slender_elements(ctx, dtype, exact):
    """Needles (a face of side h, the fourth vertex at distance 1, listed last),
    one element a row, every entry against the same inputs in higher precision.
    Rounding g_3 = -(g_0 + g_1 + g_2) twice moves it by d_3 = 2u (|g_0| + |g_1| +
    |g_2|); an entry then moves by the products with d_3 and by 8u of its terms'
    magnitudes (three products, their two sums, kw's two roundings, the
    constant, the last addition)."""
    from simit_gb300.runtime import Mesh, assemble_heat
    g = meshgen.rng(31)
    N = 4000
    h = 10 ** g.uniform(-3, 0, N)
    q = g.normal(size=(N, 3, 3))
    B = q / h[:, None, None]
    B[:, 2] = -(B[:, 0] + B[:, 1]) + g.normal(size=(N, 3))
    W, kappa, dt = g.uniform(0.5, 1, N) * 1e-3, g.uniform(0.5, 1, N) * 1e3, 1.0
    np_t = np.float32 if dtype == torch.float32 else np.float64
    B, W, kappa = (a.astype(np_t) for a in (B, W, kappa))
    mesh = Mesh(ctx, 4 * N, np.arange(4 * N, dtype=np.int32), 4)
    A, _ = assemble_heat(mesh, B.reshape(-1), W, kappa, dt, np.zeros(4 * N), dtype=dtype,
                         exact=exact)
    ctx.sync()
    got = _np(A)[:16 * N].reshape(N, 4, 4)
    up = np.float64 if dtype == torch.float32 else np.longdouble
    u = up(np.finfo(np_t).eps) / 2
    Bu, Wu = B.astype(up), W.astype(up)
    G = np.concatenate([Bu, -Bu.sum(1, keepdims=True)], 1)
    d = np.zeros_like(G)
    d[:, 3] = 2 * u * np.abs(Bu).sum(1)
    kw = (kappa.astype(up) * Wu)[:, None, None]
    mass = Wu[:, None, None] / 20 * (1 + np.eye(4, dtype=up))
    ref = mass + kw * np.einsum("nik,njk->nij", G, G)
    aG = np.abs(G)
    moved = np.einsum("nik,njk->nij", d, aG) + np.einsum("nik,njk->nij", aG, d) + \
        np.einsum("nik,njk->nij", d, d)
    bound = kw * moved + 8 * u * (mass + kw * np.einsum("nik,njk->nij", aG + d, aG + d))
    assert np.all(np.abs(got - ref) <= bound)


def _magnitudes(X, x, T, B, W):
    """Per element: n_i, the sums of |components| of the four gradients (the
    fourth from the others', as its rounding is), and f, the largest sum of
    |products| in an entry of F."""
    Ds = (x[T[:, :3]] - x[T[:, 3:]]).transpose(0, 2, 1)
    B3 = B.reshape(-1, 3, 3)
    f = np.abs(Ds) @ np.abs(B3)
    n = np.abs(B3).sum(2)
    return np.concatenate([n, n.sum(1, keepdims=True)], 1), f.max((1, 2))


@pytest.mark.parametrize("kind", ["fan", "parts", "lattice"])
@pytest.mark.parametrize("plan", [None, "gather"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_tets_entry_by_entry(ctx, oracle, kind, plan, dtype):
    """The contracted maps where the tiles change path, every entry against the
    oracle on the same rounded inputs: rows past the tile's buffers (fan), and
    11,500 vertices in random order, whose 32-row tiles hold more distinct elements
    than records and are taken in parts.  Bound: u (64 + the row's elements) of
    the entry's terms, each term's factors taken by magnitude -- a sum of that
    many terms, and for a term its products, F's rounding (4 u f in an entry of
    F, up to 20 u f + 40 u in F^-T g, log J and their products) and g_3's; twice
    that in FP64, where the oracle rounds as well."""
    from simit_gb300.runtime import (Mesh, assemble_heat, assemble_tet_force,
                                     assemble_tet_stiffness)
    if kind == "parts":
        g = meshgen.rng(12)
        mg = meshgen.tet_grid(22, 21, 22)
        X, T = mg["X0"].reshape(-1, 3), mg["tets"].reshape(-1, 4).astype(int)
        new = g.permutation(len(X))
        Y = np.empty_like(X)
        Y[new] = X
        X, T = Y, new[T][g.permutation(len(T))]
    else:
        X, T = _tets(kind)
    n, nT = len(X), len(T)
    tets = T.astype(np.int32).reshape(-1)
    np_t = np.float32 if dtype == torch.float32 else np.float64
    g = meshgen.rng(13)
    edge = min(np.linalg.norm(X[T[:, i]] - X[T[:, j]], axis=1).min()
               for i in range(4) for j in range(i))

    def inp(a):  # the values the kernels see, as float64
        return np.asarray(a, np.float64).astype(np_t).astype(np.float64)
    x = inp(X + 0.02 * edge * g.uniform(-1, 1, (n, 3)))
    v = inp(g.normal(size=n * 3))
    mu, lam = inp(g.uniform(1e3, 1e5, nT)), inp(g.uniform(1e3, 1e5, nT))
    kappa, T0 = inp(10 ** g.uniform(-2, 2, nT)), inp(g.uniform(size=n))
    c = (g.uniform(size=n) < 0.2).astype(np.int32)
    h, dt, rho, grav = 2.0 ** -7, 2.0 ** -6, 1024.0, np.array([0.125, 0.25, -9.75])
    oB, oW, _ = oracle.tet_precompute(X.reshape(-1), tets, rho)
    B, W = inp(oB), inp(oW)
    mesh = Mesh(ctx, n, tets, 4, plan=plan)
    rp, ci = mesh.pattern.host()
    sl = oracle.slots(tets, 4, rp, ci).astype(np.int64).reshape(nT, 4, 4)
    cnt = np.bincount(tets, minlength=n)
    crow = cnt[np.repeat(np.arange(n), np.diff(rp.astype(np.int64)))]
    u = float(np.finfo(np_t).eps) / 2 * (1 if dtype == torch.float32 else 2)
    mag, f = _magnitudes(X, x, T, B, W)

    def slots_of(per):  # sums of [nT, 4, 4] terms by slot
        out = np.zeros(len(ci))
        np.add.at(out, sl.reshape(-1), per.reshape(-1))
        return out

    def verts_of(per):  # sums of [nT, 4] terms by vertex
        out = np.zeros(n)
        np.add.at(out, tets, per.reshape(-1))
        return out
    nn = mag[:, :, None] * mag[:, None, :]
    mass = (0.25 * rho * W)[:, None, None] * np.eye(4)
    # heat
    A, b = assemble_heat(mesh, B, W, kappa, dt, T0, dtype=dtype, exact=False)
    oA, ob = oracle.heat_assemble(n, tets, B, W, kappa, dt, T0, rp, ci)
    ctx.sync()
    w20 = (W / 20)[:, None, None] * (1 + np.eye(4))
    bound = u * (64 + crow) * slots_of(w20 + (dt * kappa * W)[:, None, None] * nn)
    assert np.all(np.abs(_np(A) - oA) <= bound)
    bound = u * (64 + cnt) * verts_of((w20 * np.abs(T0[T])[:, None, :]).sum(2))
    assert np.all(np.abs(_np(b) - ob) <= bound)
    # elasticity, model by model
    for model in (0, 1):
        grow = 1 + (f if model else 0 * f)
        oK = oracle.tet_stiffness(model, x.reshape(-1), c, tets, B, W, mu, lam, h, rho, rp, ci)
        K = assemble_tet_stiffness(mesh, model, x.reshape(-1), c, B, W, mu, lam, h, rho,
                                   dtype=dtype, exact=False)
        ctx.sync()
        k = (h * h * W * (2 * mu + lam) * grow)[:, None, None] * nn + mass
        bound = u * (64 + crow) * slots_of(k)
        assert np.all(np.abs(_np(K).reshape(-1, 9) - oK.reshape(-1, 9)).max(1) <= bound), model
        of = oracle.tet_force(model, x.reshape(-1), v, c, tets, B, W, mu, lam, h, rho, grav)
        F = assemble_tet_force(mesh, model, x.reshape(-1), v, c, B, W, mu, lam, h, rho, grav,
                               dtype=dtype, exact=False)
        ctx.sync()
        vm = np.abs(v.reshape(n, 3)).max(1)[T]
        t = (h * W * (2 * mu + 3 * lam) * (1 + f))[:, None] * mag + \
            (0.25 * rho * W)[:, None] * (h * np.abs(grav).max() + vm)
        bound = u * (64 + cnt) * verts_of(t)
        assert np.all(np.abs(_np(F).reshape(n, 3) - of.reshape(n, 3)).max(1) <= bound), model
