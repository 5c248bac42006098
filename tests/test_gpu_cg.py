"""CG on block-tridiagonal systems with a known solution."""
import numpy as np
import pytest
import torch

from simit_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(gpu_ctx):
    return gpu_ctx


def _system(n, bs, seed=0):
    """Pattern, values (exact in FP32) and a product for a symmetric block
    tridiagonal matrix: diagonal blocks 4 I + S with |S| <= 1/4 per entry,
    off-diagonal blocks -I / 2.  Eigenvalues in [2.2, 5.8]: condition < 2.7."""
    g = np.random.default_rng(seed)
    S = g.integers(-4, 5, size=(n, bs, bs)) / 16.0
    D = np.triu(S) + np.triu(S, 1).transpose(0, 2, 1) + 4.0 * np.eye(bs)
    deg = np.full(n, 3)
    deg[0] -= 1
    deg[-1] -= 1
    rp = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    i = np.repeat(np.arange(n), deg)
    k = np.arange(rp[-1]) - rp[i]
    ci = (i + k - (i > 0)).astype(np.int32)
    vals = np.where((ci == i)[:, None, None], D[i], -0.5 * np.eye(bs))

    def mul(x):
        x = x.reshape(n, bs)
        y = np.einsum("nij,nj->ni", D, x)
        y[1:] -= 0.5 * x[:-1]
        y[:-1] -= 0.5 * x[1:]
        return y.reshape(-1)
    return rp, ci, vals.reshape(-1), mul, D


def _solver(ctx, n, bs, rp, ci, vals, dtype, **opts):
    from simit_gb300.runtime import Solver, solve_opts
    d = ctx.device
    return Solver(ctx, n, bs, torch.from_numpy(rp).to(d), torch.from_numpy(ci).to(d),
                  torch.from_numpy(vals).to(d, dtype), len(ci), solve_opts(**opts))


def test_partial_sums_of_the_right_hand_side(ctx):
    """b.b's grid is the largest of a solve's reductions here (the FP64
    product holds fewer blocks per SM); |b|^2 within 1e-13, and the solution
    within condition * tol < 1e-9 of the known one."""
    n, bs = 56000, 3
    rp, ci, vals, mul, _ = _system(n, bs)
    x0 = np.random.default_rng(1).uniform(-1, 1, n * bs)
    b = mul(x0)
    S = _solver(ctx, n, bs, rp, ci, vals, torch.float64, precision=_lib.SOLVE_F64,
                precond=_lib.PRECOND_BLOCK_JACOBI, tol=1e-10, maxiters=200)
    x = torch.zeros(n * bs, dtype=torch.float64, device=ctx.device)
    r = S.solve(torch.from_numpy(b).to(ctx.device), x)
    S.close()
    assert r.status == 1
    assert abs(r.bnorm2 - b @ b) <= 1e-13 * (b @ b)
    assert np.linalg.norm(x.cpu().numpy() - x0) <= 1e-9 * np.linalg.norm(x0)


def _pcg(mul, b, M, k):
    x, r = np.zeros_like(b), b.copy()
    z = M(r)
    p, rz = z.copy(), r @ z
    for _ in range(k):
        q = mul(p)
        a = rz / (p @ q)
        x += a * p
        r -= a * q
        z = M(r)
        rz, old = r @ z, rz
        p = z + (rz / old) * p
    return x


# around one warp's chunk of vertices (128), one chunk per SM and a second
# per warp of a block, tails of every kind, and a single row
SIZES = [1, 2, 5, 127, 129, 641, 19457, 40001]
PRECONDS = [_lib.PRECOND_NONE, _lib.PRECOND_JACOBI, _lib.PRECOND_BLOCK_JACOBI]


@pytest.mark.parametrize("iters", [1, 7, 8, 9, 24, 41])
@pytest.mark.parametrize("bs,precond", [(1, 0), (1, 1), (3, 0), (3, 1), (3, 2)])
def test_fp64_iterates(ctx, bs, precond, iters):
    """The iterate after a given number of steps (within the steps launched
    one by one, at their end, and inside graph batches) is that of the same
    recurrence in numpy.  The recurrences differ by rounding alone: at most
    41 steps * condition 2.7 * a few eps per step < 1e-12; bound 1e-11."""
    n = 1217
    rp, ci, vals, mul, D = _system(n, bs)
    b = mul(np.random.default_rng(2).uniform(-1, 1, n * bs))
    diag = np.einsum("nii->ni", D).reshape(-1)
    Di = np.linalg.inv(D)
    M = [lambda r: r.copy(), lambda r: r / diag,
         lambda r: np.einsum("nij,nj->ni", Di, r.reshape(n, bs)).reshape(-1)][precond]
    S = _solver(ctx, n, bs, rp, ci, vals, torch.float64, precision=_lib.SOLVE_F64,
                precond=PRECONDS[precond], stop=_lib.STOP_NORMR2, tol=0.0, maxiters=iters,
                verify=0)
    x = torch.zeros(n * bs, dtype=torch.float64, device=ctx.device)
    r = S.solve(torch.from_numpy(b).to(ctx.device), x)
    S.close()
    assert r.iters == iters and r.status == 2
    ref = _pcg(mul, b, M, iters)
    assert np.linalg.norm(x.cpu().numpy() - ref) <= 1e-11 * np.linalg.norm(ref)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("mixed", [0, 1])
@pytest.mark.parametrize("bs,precond", [(1, 0), (1, 1), (3, 0), (3, 1), (3, 2)])
def test_solution_at_every_size(ctx, n, mixed, bs, precond):
    """Converged solutions, from a zero start, from a guess, and with the
    guess in b's own memory (the right-hand side is overwritten by the
    solution): within condition * tol < 1e-9 of the known one."""
    rp, ci, vals, mul, _ = _system(n, bs, seed=n)
    d = ctx.device
    x0 = np.random.default_rng(3).uniform(-1, 1, n * bs)
    b = torch.from_numpy(mul(x0)).to(d)
    S = _solver(ctx, n, bs, rp, ci, vals, torch.float32 if mixed else torch.float64,
                precision=_lib.SOLVE_MIXED if mixed else _lib.SOLVE_F64,
                precond=PRECONDS[precond], tol=1e-10, maxiters=200)
    guess = torch.from_numpy(x0 + 0.1 * np.cos(np.arange(n * bs))).to(d)
    own = b.clone()
    runs = [(S.solve_ex(b, (z := torch.full_like(b, 7.0)), x_zero=True), z),
            (S.solve(b, guess), guess), (S.solve(own, own), own)]
    S.close()
    for r, x in runs:
        assert r.status == 1
        assert np.linalg.norm(x.cpu().numpy() - x0) <= 1e-9 * np.linalg.norm(x0)


@pytest.mark.parametrize("mixed", [0, 1])
@pytest.mark.parametrize("precond", [0, 1, 2])
def test_breakdown_then_a_solve(ctx, mixed, precond):
    """A negative definite matrix stops at p.q < 0 with status 3; the same
    solver, with the matrix negated in place, then converges."""
    n, bs = 641, 3
    rp, ci, vals, mul, _ = _system(n, bs)
    d = ctx.device
    dt = torch.float32 if mixed else torch.float64
    from simit_gb300.runtime import Solver, solve_opts
    v = torch.from_numpy(-vals).to(d, dt)
    S = Solver(ctx, n, bs, torch.from_numpy(rp).to(d), torch.from_numpy(ci).to(d), v, len(ci),
               solve_opts(precision=_lib.SOLVE_MIXED if mixed else _lib.SOLVE_F64,
                          precond=PRECONDS[precond], tol=1e-10, maxiters=200))
    x0 = np.random.default_rng(4).uniform(-1, 1, n * bs)
    b = torch.from_numpy(mul(x0)).to(d)
    assert S.solve(b, torch.zeros_like(b)).status == 3
    v.neg_()
    S.refresh()
    x = torch.zeros_like(b)
    assert S.solve(b, x).status == 1
    S.close()
    assert np.linalg.norm(x.cpu().numpy() - x0) <= 1e-9 * np.linalg.norm(x0)


@pytest.mark.parametrize("bs,opts", [
    (1, dict(precision=_lib.SOLVE_MIXED, precond=_lib.PRECOND_JACOBI, lanes=-10)),
    (3, dict(precision=_lib.SOLVE_MIXED, precond=_lib.PRECOND_BLOCK_JACOBI)),
    (3, dict(precision=_lib.SOLVE_MIXED, precond=_lib.PRECOND_BLOCK_JACOBI, lanes=-2)),
    (3, dict(precision=_lib.SOLVE_MIXED, precond=_lib.PRECOND_BLOCK_JACOBI, storage=1, wide=40)),
    (3, dict(precision=_lib.SOLVE_F64, precond=_lib.PRECOND_BLOCK_JACOBI))])
def test_two_matrices_in_turn(ctx, bs, opts):
    """A matrix with long rows and one with short rows, whose products stage
    tiles of different sizes, solved in turn by solvers that both live."""
    d, n = ctx.device, 5000
    opts = dict(opts)
    wide = opts.pop("wide", 90)  # a dense leading block: rows this long
    rp, ci, vals, mul, _ = _system(n, bs)
    import scipy.sparse as sp
    A = sp.bsr_matrix((vals.reshape(-1, bs, bs), ci, rp)).tocsr()
    W = sp.kron(sp.csr_matrix((np.full((wide, wide), 1 / 64.0).reshape(-1),
                               (np.repeat(np.arange(wide), wide), np.tile(np.arange(wide), wide))),
                              shape=(n, n)), sp.identity(bs)).tocsr()
    out = []
    for M in (A + W, A):
        B = M.tobsr((bs, bs))
        B.sort_indices()
        S = _solver(ctx, n, bs, B.indptr.astype(np.int32), B.indices.astype(np.int32),
                    np.ascontiguousarray(B.data).reshape(-1),
                    torch.float32 if opts["precision"] == _lib.SOLVE_MIXED else torch.float64,
                    tol=1e-10, maxiters=300, **opts)
        out.append((S, M))
    x0 = np.random.default_rng(5).uniform(-1, 1, n * bs)
    for S, M in out + out[::-1]:
        b = torch.from_numpy(M @ x0).to(d)
        x = torch.zeros_like(b)
        assert S.solve(b, x).status == 1
        assert np.linalg.norm(x.cpu().numpy() - x0) <= 1e-9 * np.linalg.norm(x0)
    for S, _ in out:
        S.close()
