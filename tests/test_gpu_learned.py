"""GPU checks of the learned preconditioner: forward and backward against the
numpy oracle (oracle/mpnn_oracle.py), training, and its use in flexible PCG."""
import os

import numpy as np
import pytest
import torch

from simit_gb300 import _lib, problems

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(gpu_ctx):
    return gpu_ctx


def _small(ctx, ncell=4, seed=3):
    host = problems.hetero_mesh(ncell, seed=seed)
    return problems.HeteroElasticity(ctx, host, dtype=torch.float32,
                                     precond=_lib.PRECOND_BLOCK_JACOBI)


@pytest.mark.parametrize("form", ["relu", "linear", "sym"])
def test_forward_backward_match_oracle(ctx, form):
    from oracle import mpnn_oracle as mo
    from simit_gb300 import learned
    prob = _small(ctx, 4)
    m = prob.mesh
    rp, ci = m.pattern.host()
    vals = prob.A.cpu().numpy()
    g = learned.Graph(ctx, m, prob.A, form=form)
    params = learned.init_params(seed=5, out_scale=1.0)
    rng = np.random.Generator(np.random.Philox(11))
    r = rng.normal(size=m.n * 3).astype(np.float32)
    dz = rng.normal(size=m.n * 3).astype(np.float32)
    d = ctx.device
    pt = torch.tensor(params, device=d)
    rt = torch.tensor(r, device=d)
    zt = torch.empty_like(rt)
    g.forward(pt, rt, zt, train=True)
    grad = torch.zeros_like(pt)
    g.backward(pt, torch.tensor(dz, device=d), grad)
    if form == "sym":
        z_ref, cache = mo.forward_sym(params, m.n, rp, ci, vals, r)
        gref = mo.backward_sym(cache, dz)
        s = np.einsum("vij,vj->vi", mo.block_jacobi(m.n, rp, ci, vals),
                      r.reshape(-1, 3).astype(np.float64)).reshape(-1)
    else:
        z_ref, cache = mo.forward(params, m.n, rp, ci, vals, r, linear=form == "linear")
        gref = mo.backward(cache, dz)
        s = cache["s"].reshape(-1)
    z = zt.cpu().numpy()
    # FP32 accumulation vs FP64 (bf16 operands rounded identically up to
    # ties flipped by the accumulation order)
    assert np.linalg.norm(z - z_ref) <= 1e-3 * np.linalg.norm(z_ref - s) + 1e-6 * np.linalg.norm(s)
    gg = grad.cpu().numpy()
    o = 0
    for name, (a, b) in mo.SHAPES:
        seg = slice(o, o + a * b)
        o += a * b
        err = np.linalg.norm(gg[seg] - gref[seg])
        assert err <= 2e-3 * np.linalg.norm(gref[seg]) + 1e-6, (name, err, np.linalg.norm(gref[seg]))
    g.close()
    prob.close()


@pytest.mark.parametrize("form", ["relu", "linear", "sym"])
@pytest.mark.parametrize("ncell", [2, 3, 7, 9])
def test_backward_at_tile_edges(ctx, form, ncell):
    """27, 64, 512 and 1,000 vertices: below, at and past the backward's
    tiles of 64 vertices and slabs of 32.  The bound is the one above: the
    oracle sums in FP64 what the kernels sum in FP32."""
    from oracle import mpnn_oracle as mo
    from simit_gb300 import learned
    prob = _small(ctx, ncell)
    m = prob.mesh
    rp, ci = m.pattern.host()
    vals = prob.A.cpu().numpy()
    g = learned.Graph(ctx, m, prob.A, form=form)
    params = learned.init_params(seed=6, out_scale=1.0)
    rng = np.random.Generator(np.random.Philox(ncell))
    r, dz = rng.normal(size=(2, m.n * 3)).astype(np.float32)
    d = ctx.device
    pt, rt = torch.tensor(params, device=d), torch.tensor(r, device=d)
    zt, grad = torch.empty_like(rt), torch.full_like(pt, float("nan"))
    g.forward(pt, rt, zt, train=True)
    g.backward(pt, torch.tensor(dz, device=d), grad)
    if form == "sym":
        gref = mo.backward_sym(mo.forward_sym(params, m.n, rp, ci, vals, r)[1], dz)
    else:
        gref = mo.backward(mo.forward(params, m.n, rp, ci, vals, r, linear=form == "linear")[1], dz)
    gg, o = grad.cpu().numpy(), 0
    for name, (a, b) in mo.SHAPES:
        seg = slice(o, o + a * b)
        o += a * b
        err = np.linalg.norm(gg[seg] - gref[seg])
        assert err <= 2e-3 * np.linalg.norm(gref[seg]) + 1e-6, (name, err, np.linalg.norm(gref[seg]))
    g.close()
    prob.close()


@pytest.mark.parametrize("form", ["relu", "sym"])
def test_training_reduces_loss(ctx, form):
    from simit_gb300 import learned
    prob, pairs = learned.make_pairs(ctx, 6, seed=21, n_rhs=2, ks=(4, 16, 64))
    g = learned.Graph(ctx, prob.mesh, prob.A, form=form)
    tr = learned.Trainer(ctx, lr=3e-3, seed=1)
    L0 = tr.eval_loss(g, pairs)
    for _ in range(40):
        for r, e, eAe in pairs:
            tr.step(g, r, e, eAe)
    L1 = tr.eval_loss(g, pairs)
    # the symmetric form starts at block Jacobi (Wout = 0), already a good
    # single-step operator, and has less to gain on a 6^3 mesh
    assert L1 < (0.95 if form == "relu" else 0.97) * L0, (L0, L1)
    g.close()
    prob.close()


def test_learned_fpcg_converges_and_falls_back(ctx):
    from simit_gb300 import learned
    res = learned.compare(ctx, learned.init_params(seed=2, out_scale=0.01), 8)
    assert res["learned"]["status"] == 1 and res["learned"]["relres"] <= 1e-8
    bad = learned.init_params(seed=2, out_scale=1.0)
    bad[-1] = np.nan  # a NaN output weight poisons z: the solver falls back
    res = learned.compare(ctx, bad, 8)
    assert res["learned"]["fallbacks"] >= 1
    assert res["learned"]["status"] == 1 and res["learned"]["relres"] <= 1e-8


@pytest.mark.parametrize("form", ["relu", "linear", "sym"])
def test_trained_network_gain(ctx, form):
    """What the committed trained weights gain over block-Jacobi PCG (the
    method without the network) on a held-out 24^3 mesh, to the same FP64
    residual, printed for every form.  The relu and linear forms are not
    symmetric operators and lose to block Jacobi inside PCG (recorded, not
    asserted); the symmetric factorized form must take fewer iterations."""
    from simit_gb300 import learned
    if not os.path.exists(learned.WEIGHTS[form]):
        pytest.skip("no trained weights committed for " + form)
    res = learned.compare(ctx, learned.load_weights(form), 24, seed=777, form=form)
    bj, ln = res["block_jacobi"], res["learned"]
    print("%s: learned %d iters %.1f ms, block-Jacobi %d iters %.1f ms, iteration gain %.2fx"
          % (form, ln["iters"], ln["ms"], bj["iters"], bj["ms"], bj["iters"] / ln["iters"]))
    assert bj["status"] == 1 and ln["status"] == 1
    assert ln["relres"] <= 1e-8
    if form == "sym":
        assert ln["fallbacks"] == 0
        assert ln["iters"] < bj["iters"]


def test_folded_forward_matches_layered_and_oracle(ctx):
    """The symmetric form evaluated as its degree-6 matrix polynomial (six
    Horner gather passes) against the oracle's restatement in FP64: in FP32,
    and with FP16 edge weights and block-floating-point vectors (the oracle
    rounding at the same points); and against the tensor-core layered
    evaluation of the same network."""
    from oracle import mpnn_oracle as mo
    from simit_gb300 import learned
    prob = _small(ctx, 6, seed=5)
    m = prob.mesh
    rp, ci = m.pattern.host()
    vals = prob.A.cpu().numpy()
    g = learned.Graph(ctx, m, prob.A, form="sym")
    params = learned.load_weights("sym")
    rng = np.random.Generator(np.random.Philox(12))
    r = rng.normal(size=m.n * 3).astype(np.float32)
    d = ctx.device
    pt = torch.tensor(params, device=d)
    rt = torch.tensor(r, device=d)
    out = {}
    for mode in (_lib.MPNN_EXEC_FOLDED_F32, _lib.MPNN_EXEC_FOLDED, _lib.MPNN_EXEC_LAYERED):
        g.set_exec(mode)
        zt = torch.empty_like(rt)
        g.forward(pt, rt, zt)
        ctx.sync()
        out[mode] = zt.cpu().numpy().astype(np.float64)
    z_ref = mo.forward_sym_poly(params, m.n, rp, ci, vals, r)
    a, _, _ = mo.edge_weights(m.n, rp, ci, vals)
    # the FP16 evaluation: FP16 edge weights and block-floating-point vectors
    z_ref16 = mo.forward_sym_poly(params, m.n, rp, ci, vals, r,
                                    a=a.astype(np.float16).astype(np.float64), bfp=True)
    bj = np.einsum("vij,vj->vi", mo.block_jacobi(m.n, rp, ci, vals),
                   r.reshape(-1, 3).astype(np.float64)).reshape(-1)
    corr = np.linalg.norm(z_ref - bj)
    assert corr > 1e-3 * np.linalg.norm(bj)
    e32 = np.linalg.norm(out[_lib.MPNN_EXEC_FOLDED_F32] - z_ref)
    e16 = np.linalg.norm(out[_lib.MPNN_EXEC_FOLDED] - z_ref16)
    el = np.linalg.norm(out[_lib.MPNN_EXEC_LAYERED] - out[_lib.MPNN_EXEC_FOLDED_F32])
    print("folded FP32 %.2e, folded FP16 %.2e, layered vs folded %.2e (of the correction %.3e)"
          % (e32 / corr, e16 / corr, el / corr, corr))
    # FP32 arithmetic (FP32 folded matrices and sums) against FP64
    assert e32 <= 2e-5 * corr
    assert e16 <= 2e-4 * corr
    # the layered kernels carry the hidden layers as split bf16 (about 2^-16)
    assert el <= 1e-3 * corr
    g.close()
    prob.close()


def test_folded_solve_matches_layered_solve(ctx):
    """Flexible PCG with the folded evaluation takes the iterations of the
    layered one (the same operator) and converges to the FP64 tolerance."""
    from simit_gb300 import learned
    w = learned.load_weights("sym")
    rf = learned.compare(ctx, w, 12, seed=778)
    rl = learned.compare(ctx, w, 12, seed=778, exec_mode=_lib.MPNN_EXEC_LAYERED)
    ff, ll = rf["learned"], rl["learned"]
    print("folded %d iters %.1f ms, layered %d iters %.1f ms" % (ff["iters"], ff["ms"],
                                                                 ll["iters"], ll["ms"]))
    assert ff["status"] == 1 and ff["relres"] <= 1e-8 and ff["fallbacks"] == 0
    assert abs(ff["iters"] - ll["iters"]) <= max(2, 0.03 * ll["iters"])


@pytest.mark.parametrize("mode", [_lib.MPNN_EXEC_FOLDED, _lib.MPNN_EXEC_FOLDED_F32])
def test_folded_forward_long_rows(ctx, mode):
    """A pattern with one row of 5000 entries (a vertex joined to every
    other one) beside rows of 2-3: the Horner passes' lanes loop over the
    long row; the result matches the oracle's polynomial (FP16 evaluation:
    with the oracle rounding where the GPU stores)."""
    from oracle import mpnn_oracle as mo
    from simit_gb300 import learned
    from simit_gb300.runtime import Mesh
    n = 5000
    edges = np.array([(0, i) for i in range(1, n)] + [(i, i + 1) for i in range(1, n - 1)],
                     dtype=np.int32)
    m = Mesh(ctx, n, edges, 2)
    rp, ci = m.pattern.host()
    rows = np.repeat(np.arange(n), np.diff(rp.astype(np.int64)))
    rng = np.random.Generator(np.random.Philox(13))
    blocks = rng.normal(0, 0.1, size=(m.nnzb, 3, 3))
    diag = rows == ci.astype(np.int64)
    S = rng.normal(0, 0.2, size=(int(diag.sum()), 3, 3))
    blocks[diag] = 10.0 * np.eye(3) + 0.5 * (S + np.transpose(S, (0, 2, 1)))
    vals = blocks.reshape(-1).astype(np.float32)
    A = torch.tensor(vals, device=ctx.device)
    g = learned.Graph(ctx, m, A, form="sym")
    g.set_exec(mode)
    params = learned.load_weights("sym")
    r = rng.normal(size=n * 3).astype(np.float32)
    pt = torch.tensor(params, device=ctx.device)
    rt = torch.tensor(r, device=ctx.device)
    zt = torch.empty_like(rt)
    g.forward(pt, rt, zt)
    ctx.sync()
    a, _, _ = mo.edge_weights(n, rp, ci, vals.astype(np.float64))
    half = mode == _lib.MPNN_EXEC_FOLDED
    z_ref = mo.forward_sym_poly(params, n, rp, ci, vals.astype(np.float64), r,
                                a=a.astype(np.float16).astype(np.float64) if half else a,
                                bfp=half)
    err = np.linalg.norm(zt.cpu().numpy() - z_ref)
    assert err <= 1e-5 * np.linalg.norm(z_ref), err
    g.close()


@pytest.mark.parametrize("mode", [_lib.MPNN_EXEC_FOLDED, _lib.MPNN_EXEC_FOLDED_F32])
@pytest.mark.parametrize("ncell", [1, 4, 16, 36, 50, 51])
def test_learned_solve_at_grid_edges(ctx, ncell, mode):
    """Learned solves around the sizes where the iteration's one launch
    changes shape: fewer slices of 32 rows than SMs, two warps per SM, more
    than 8, the 28 it can hold, and one more than that (separate kernels).
    Each reaches the verified tolerance without falling back, twice with the
    same bits; the FP32 evaluation, the layered one's operator, in its number
    of iterations at the small sizes."""
    from simit_gb300 import learned
    from simit_gb300.runtime import Solver, solve_opts
    w = learned.load_weights("sym")
    host = problems.reorder_hetero(problems.hetero_mesh(ncell, seed=5))
    prob = problems.HeteroElasticity(ctx, host, dtype=torch.float32,
                                     precond=_lib.PRECOND_BLOCK_JACOBI)
    m = prob.mesh
    wt = torch.tensor(np.asarray(w, np.float32), device=ctx.device)
    b = torch.randn(m.n * 3, dtype=torch.float64, generator=torch.Generator().manual_seed(7))
    b = b.to(ctx.device)
    torch.cuda.synchronize()

    def solve(exec_mode):
        S = Solver(ctx, m.n, 3, m.pattern.rowptr, m.pattern.colidx, prob.A, m.nnzb,
                   solve_opts(precision=_lib.SOLVE_MIXED, precond=_lib.PRECOND_LEARNED, tol=1e-8,
                              maxiters=5000, learned_params=wt,
                              learned_form=learned.FORMS["sym"], learned_exec=exec_mode),
                   learned_params_keep=wt)
        out = []
        for _ in range(2):
            x = torch.zeros_like(b)
            torch.cuda.synchronize()
            r = S.solve(b, x)
            assert r.status == 1 and r.fallbacks == 0
            assert r.true_normr2 <= 1e-16 * r.bnorm2
            out.append((x, r.iters))
        S.close()
        assert torch.equal(out[0][0], out[1][0])
        return out[0][1]
    it = solve(mode)
    if ncell <= 16 and mode == _lib.MPNN_EXEC_FOLDED_F32:
        assert abs(it - solve(_lib.MPNN_EXEC_LAYERED)) <= max(2, 0.03 * it)
    prob.close()
