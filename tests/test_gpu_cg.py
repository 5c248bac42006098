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
