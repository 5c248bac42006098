"""GPU checks of the batched PCG (many uneven cloth sheets in one launch)."""
import ctypes

import numpy as np
import pytest
import torch

from simit_gb300 import _lib, problems

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(gpu_ctx):
    return gpu_ctx


@pytest.fixture(scope="module")
def batch(ctx):
    host = problems.cloth_batch(nsheets=12, lo=8, hi=40, seed=3)
    return problems.ClothBatch(ctx, host)


def test_every_sheet_converges_on_the_true_residual(ctx, batch, oracle):
    batch.step()
    ctx.sync()
    st = batch.status.cpu().numpy()
    assert np.all(st == 1), st
    assert np.all(batch.relres.cpu().numpy() <= 1e-6)
    # independent check: each sheet's FP64 residual with the oracle SpMV
    rp, ci = batch.mesh.pattern.host()
    A = batch.A.cpu().numpy().astype(np.float64)
    f = batch.f.cpu().numpy().astype(np.float64)
    v = batch.vout.cpu().numpy().astype(np.float64)
    r = f - oracle.spmv(batch.mesh.n, 3, rp, ci, A, v)
    sp = batch.host["sys_ptr"]
    for s in range(batch.nsys):
        a, b = sp[s] * 3, sp[s + 1] * 3
        assert np.linalg.norm(r[a:b]) <= 1.001e-6 * np.linalg.norm(f[a:b]), s


def test_matches_one_at_a_time_solves(ctx, batch):
    """Each sheet solved alone by the general mixed-precision solver reaches
    the same solution (both to a 1e-6 relative residual)."""
    from simit_gb300.runtime import Mesh, Solver, assemble_springs, solve_opts
    batch.step()
    ctx.sync()
    vb = batch.vout.cpu().numpy()
    h = batch.host
    sp = h["sys_ptr"]
    ep = h["ep"].reshape(-1, 2)
    for s in range(batch.nsys):
        v0, v1 = sp[s], sp[s + 1]
        sel = (ep[:, 0] >= v0) & (ep[:, 0] < v1)
        mesh = Mesh(ctx, int(v1 - v0), (ep[sel] - v0).reshape(-1), 2)
        c = problems.CLOTH
        A, f = assemble_springs(mesh, h["x"][v0 * 3:v1 * 3], np.zeros((v1 - v0) * 3),
                                np.full(v1 - v0, c["mass"]), h["fixed"][v0:v1], h["k"][sel],
                                h["l0"][sel], c["dt"], c["viscous"], c["grav"], form=0,
                                dtype=torch.float32, exact=False)
        S = Solver(ctx, mesh.n, 3, mesh.pattern.rowptr, mesh.pattern.colidx, A, mesh.nnzb,
                   solve_opts(precision=_lib.SOLVE_MIXED, precond=_lib.PRECOND_BLOCK_JACOBI,
                              tol=1e-6, maxiters=10000))
        x = torch.zeros(mesh.n * 3, dtype=torch.float64, device=ctx.device)
        res = S.solve(f.double(), x)
        S.close()
        assert res.status == 1
        xs = x.cpu().numpy()
        assert np.linalg.norm(xs - vb[v0 * 3:v1 * 3]) <= 1e-4 * np.linalg.norm(xs)


def test_graph_replay_is_deterministic(ctx, batch):
    batch.capture()
    batch.replay()
    ctx.sync()
    v1 = batch.vout.clone()
    batch.replay()
    ctx.sync()
    assert torch.equal(v1, batch.vout)
    assert 0 <= batch.config < _lib.load().sg_batched_configs()


GRID_CONFIGS = (6, 7)  # the whole grid on all systems


@pytest.mark.parametrize("sides", [[2], [8], [3, 9, 33, 8], [2] * 400 + [5, 70], [64, 100]])
def test_grid_wide_matches_per_system(ctx, sides):
    """The grid-wide schedule against the per-system one: one tiny system,
    systems of exactly a chunk, more systems than a CTA keeps in shared
    memory, systems over many CTAs -- same status, and the same solution as
    far as two solves to a 1e-6 residual agree (1e-4, as above)."""
    parts, off = [], 0
    from simit_gb300 import meshgen
    g = meshgen.rng(4)
    for s in sides:
        sh = meshgen.cloth_sheet(s)
        x = sh["x"].reshape(-1, 3).copy()
        x[:, 2] += g.uniform(-0.2, 0.2, len(x)) / (s - 1)
        parts.append((x.reshape(-1), sh["ep"] + off, np.where(sh["is_bend"] > 0, 50.0, 5e3),
                      sh["l0"], sh["fixed"]))
        off += sh["n"]
    x, ep, k, l0, fixed = [np.concatenate(t) for t in zip(*parts)]
    host = {"n": off, "x": x, "ep": ep.astype(np.int32), "k": k, "l0": l0, "fixed": fixed,
            "sys_ptr": np.concatenate([[0], np.cumsum(np.square(sides))]).astype(np.int32),
            "sides": np.asarray(sides)}
    cb = problems.ClothBatch(ctx, host, config=3)
    cb.step()
    ctx.sync()
    ref, st = cb.vout.cpu().numpy(), cb.status.cpu().numpy()
    for cfg in GRID_CONFIGS:
        cb.step(config=cfg)
        ctx.sync()
        assert np.array_equal(cb.status.cpu().numpy(), st)
        assert np.all(cb.relres.cpu().numpy()[st == 1] <= 1e-6)
        v = cb.vout.cpu().numpy()
        assert np.linalg.norm(v - ref) <= 1e-4 * np.linalg.norm(ref)
        first = cb.vout.clone()
        cb.step(config=cfg)
        ctx.sync()
        assert torch.equal(first, cb.vout)
    # the iteration limit: stopped after as many iterations, with its status
    for maxiters in (0, 5):
        cb.step(config=3, maxiters=maxiters)
        ctx.sync()
        st, it = cb.status.cpu().numpy(), cb.iters.cpu().numpy()
        for cfg in GRID_CONFIGS:
            cb.step(config=cfg, maxiters=maxiters)
            ctx.sync()
            assert np.array_equal(cb.status.cpu().numpy(), st)
            assert np.array_equal(cb.iters.cpu().numpy(), it)


def test_grid_wide_systems_without_rows(ctx):
    """Empty systems among the others finish at once, converged."""
    host = problems.cloth_batch(nsheets=3, lo=6, hi=20, seed=9)
    sp = host["sys_ptr"]
    host = dict(host, sys_ptr=np.array([0, 0, sp[1], sp[1], sp[1], sp[2], sp[3], sp[3]], np.int32))
    cb = problems.ClothBatch(ctx, host, config=3)
    cb.step()
    ctx.sync()
    st, it = cb.status.cpu().numpy(), cb.iters.cpu().numpy()
    assert np.all(st == 1)
    for cfg in GRID_CONFIGS:
        cb.step(config=cfg)
        ctx.sync()
        assert np.array_equal(cb.status.cpu().numpy(), st)
        assert np.all(cb.iters.cpu().numpy()[it == 0] == 0)


def test_grid_wide_systems_over_many_ctas_repeat(ctx):
    """Systems whose rows belong to many CTAs, with small ones between them so
    that the CTAs of one system have unequal work: every run takes the same
    decisions on every system (equal bits, iterations and statuses)."""
    host = problems.cloth_batch(nsheets=40, lo=8, hi=120, seed=17)
    cb = problems.ClothBatch(ctx, host, config=3)
    for cfg in GRID_CONFIGS:
        first = None
        for _ in range(12):
            cb.step(config=cfg)
            ctx.sync()
            got = [t.clone() for t in (cb.vout, cb.iters, cb.status, cb.relres)]
            assert bool((cb.status == 1).all()) and float(cb.relres.max()) <= 1e-6
            first = first or got
            assert all(torch.equal(a, b) for a, b in zip(first, got))


def test_every_config_takes_unaligned_arrays(ctx):
    """Values and columns that start one element past a 16-byte boundary: every
    configuration solves every system, to the solution of the aligned arrays
    (1e-4, as two solves to a 1e-6 residual agree above)."""
    from simit_gb300.runtime import call, ptr
    host = problems.cloth_batch(nsheets=5, lo=6, hi=70, seed=23)
    cb = problems.ClothBatch(ctx, host, config=3)
    cb.step()
    ctx.sync()
    ref = cb.vout.clone()
    nnzb = cb.mesh.nnzb
    with ctx.stream():
        vals = torch.empty(nnzb * 9 + 1, dtype=torch.float32, device=ctx.device)[1:]
        cols = torch.empty(nnzb + 1, dtype=torch.int32, device=ctx.device)[1:]
        vals.copy_(cb.A[:nnzb * 9])
        cols.copy_(cb.mesh.pattern.colidx[:nnzb].view(torch.int32))
    assert vals.data_ptr() % 16 and cols.data_ptr() % 16
    A = _lib.Matrix(cb.mesh.n, 3, nnzb, cb.mesh.pattern.rowptr.data_ptr(), cols.data_ptr(),
                    _lib.F32, vals.data_ptr())
    for cfg in range(_lib.load().sg_batched_configs()):
        with ctx.stream():
            x = cb.v.clone()
        call("sg_batched_pcg", ctx.h, cb.nsys, ptr(cb.sys_ptr), ptr(cb.order), ctypes.byref(A),
             ptr(cb.f), ptr(x), problems.CLOTH["tol"], 10000, cfg, ptr(cb.iters), ptr(cb.status),
             ptr(cb.relres))
        ctx.sync()
        assert bool((cb.status == 1).all()) and float(cb.relres.max()) <= 1e-6, cfg
        assert float((x - ref).norm()) <= 1e-4 * float(ref.norm()), cfg
