"""Branches that only some inputs reach: the eigensolvers behind the SVD start
and the row sums of the batched CP-ALS."""
import numpy as np
import pytest

import tenrso_b200 as tb

pytestmark = pytest.mark.gpu


def unfold(X, m):
    return np.moveaxis(X.astype(np.float64), m, 0).reshape(X.shape[m], -1)


# tridiagonalisation up to 160 rows, Jacobi rotations beyond and where leading
# eigenvalues coincide; one row, more columns asked for than rows of the Gram
# are independent
@pytest.mark.parametrize("kind,shape,R", [
    ("normal", (160, 9, 31), 16), ("normal", (161, 9, 31), 16), ("normal", (33, 2, 40), 2),
    ("normal", (1, 12, 30), 1), ("equal", (24, 24, 1), 6), ("rank1", (40, 21, 17), 1),
    ("huge", (20, 30, 11), 5), ("tiny", (20, 30, 11), 5)])
def test_svd_start(kind, shape, R):
    """Each factor column is a unit eigenvector of X_(n) X_(n)^T: FP64 vectors
    rounded to FP32 (6e-8 per entry), so the residual is at most 1e-6 of the
    largest eigenvalue and the columns are orthonormal to 1e-6; the values are
    the leading ones to 1e-6."""
    rng = np.random.default_rng(len(kind) + sum(shape))
    if kind == "equal":  # an orthogonal matrix: every singular value is 1
        X = np.linalg.qr(rng.standard_normal(shape[:2]))[0].reshape(shape)
    elif kind == "rank1":
        X = np.einsum("i,j,k->ijk", *[rng.standard_normal(n) for n in shape])
    else:
        X = rng.standard_normal(shape) * {"normal": 1.0, "huge": 1e15, "tiny": 1e-15}[kind]
    X = X.astype(np.float32)
    for m, F in enumerate(tb.initialize_factors(X, R, "svd", seed=3)):
        G = unfold(X, m) @ unfold(X, m).T
        lam = np.linalg.eigvalsh(G)[::-1]
        F = F.astype(np.float64)
        k = min(R, shape[m], X.size // shape[m])
        V = F[:, :k]
        assert np.abs(V.T @ V - np.eye(k)).max() <= 1e-6, m
        val = np.einsum("ir,ij,jr->r", V, G, V)
        assert np.abs(val - lam[:k]).max() <= 1e-6 * lam[0], m
        assert np.linalg.norm(G @ V - V * val, axis=0).max() <= 1e-6 * lam[0], m


@pytest.mark.parametrize("threads,cps", [(128, 4), (256, 2), (512, 1)])
@pytest.mark.parametrize("long", [0, 5900])
def test_batched_row_sums(orc, threads, cps, long):
    """Items that meet in shared memory, and (with an instance that fills it)
    atomic sums; several groups per row, rows that straddle a block of items,
    one-element modes. The fit after ten sweeps to 1e-4 of the FP64 one."""
    shapes = [((5, 4, 3), 2), ((2, 70, 90), 2), ((40, 3, 17), 3), ((96, 33, 61), 16),
              ((1, 9, 30), 1)] + ([((4, long, 8), 4)] if long else [])
    rng = np.random.default_rng(9)
    Xs, inits = [], []
    for s, R in shapes:
        fs = [rng.random((n, R)) + 0.1 for n in s]
        X = np.einsum("ir,jr,kr->ijk", *fs)
        X += 0.05 * np.linalg.norm(X) / np.sqrt(X.size) * rng.standard_normal(s)
        Xs.append(X.astype(np.float32))
        inits.append([rng.random((n, R)).astype(np.float32) for n in s])
    b = tb.BatchedCpAls(Xs, [R for _, R in shapes])
    b.set_config(threads, 0, cps)
    for X, (s, R), init, r in zip(Xs, shapes, inits, b.cp_als(10, 0.0, init=inits)):
        _, info = orc.cp_als(X.astype(np.float64), R, 10, 0.0,
                             [f.astype(np.float64) for f in init])
        assert r.iters == info["iters"]
        assert abs(r.fit - info["fit"]) <= 1e-4, (s, R)
    b.close()


# the stop decision is taken beside the next sweep's first MTTKRP, and the host
# looks at it every eighth sweep: stops at sweeps 3, 20, 33, 8 and 13
@pytest.mark.parametrize("shape,R,tol", [((70, 40, 33), 5, 2e-2), ((70, 40, 33), 5, 3e-3),
                                         ((70, 40, 33), 5, 3e-4), ((20, 16, 12, 9), 4, 1e-2),
                                         ((20, 16, 12, 9), 4, 3e-3)])
def test_cp_als_f64_stops(orc, shape, R, tol):
    """The sweeps enqueued past a stop leave factors, fit and history as they
    are. FP64 on both sides: factors to 1e-6, the history to 1e-9, as in the
    other FP64 CP-ALS tests."""
    from tenrso_b200 import synth
    X, _ = synth.dense_lowrank(shape, R, seed=0xF6, dist="uniform", noise=0.01,
                               dtype=np.float64)
    init = [synth.uniform(0xF6, 200 + m, (n, R)) for m, n in enumerate(shape)]
    res = tb.cp_als_f64(X, R, 60, tol, init=init)
    U, info = orc.cp_als(X, R, 60, tol, init)
    assert res.iters == info["iters"] and res.convergence.reason == info["reason"]
    assert np.abs(res.convergence.fit_history - info["fit_history"]).max() <= 1e-9
    for a, b in zip(res.factors, U):
        assert np.linalg.norm(a - b) <= 1e-6 * np.linalg.norm(b)


# BF16x3 CP-ALS off the single-layout path: bf16 unfoldings and the tensor-core
# kernels on them. One element into its buffer, a tensor of any shape runs so;
# aligned, long or high-rank three-mode tensors do (all unfoldings in one pass).
# Run-scaled kernel: run lengths 8..384, padded k-blocks, odd ranks, several
# runs per CTA, 4-way weights; (129, 70, 31) and (8, 9, 10, 3, 4): the other one.
@pytest.mark.parametrize("shape,R,offset", [
    ((130, 5, 192), 5, 1), ((70, 6, 4, 128), 4, 1), ((40, 7, 384), 7, 1), ((300, 64, 64), 16, 1),
    ((33, 12, 3, 64), 3, 1), ((70, 6, 48), 6, 1), ((16, 12, 8, 48), 8, 1), ((50, 9, 104), 9, 1),
    ((24, 40, 8), 5, 1), ((129, 70, 31), 20, 1), ((8, 9, 10, 3, 4), 3, 1), ((80, 72, 88), 70, 1),
    ((128, 1024, 64), 8, 0), ((80, 72, 88), 70, 0), ((90, 33, 20), 17, 0)])
def test_cp_als_bf16x3_unfoldings(shape, R, offset):
    """One sweep against FP64. An MTTKRP is good to 1e-5 of its norm (BF16x3
    keeps 16 bits of each factor of a product, and the errors average), and each
    solve multiplies the errors so far by at most the condition of its normal
    equations; ten times that, once per mode."""
    import torch
    rng = np.random.default_rng(sum(shape) + R)
    X = rng.standard_normal(shape).astype(np.float32)
    init = [rng.standard_normal((n, R)).astype(np.float32) for n in shape]
    buf = torch.empty(X.size + offset, device="cuda")
    buf[offset:].copy_(torch.from_numpy(X.ravel()))
    d_init = torch.from_numpy(np.concatenate([f.ravel() for f in init])).cuda()
    out = torch.empty_like(d_init)
    torch.cuda.synchronize()
    ctx, launches = tb.Context(), {}
    for precision in ("fp32", "bf16x3"):
        before = ctx.launches
        tb.cp_als_dev(buf.data_ptr() + 4 * offset, shape, R, 1, 0.0, d_init.data_ptr(),
                      out.data_ptr(), precision, ctx=ctx)
        launches[precision] = ctx.launches - before
    one_pass = offset == 0 and shape[1] % 8 == 0 and shape[2] % 8 == 0  # with the norm of X
    assert launches["bf16x3"] - launches["fp32"] == (0 if one_pass else len(shape))
    got, off, bound = out.cpu().numpy(), 0, 0.0
    fs = [f.astype(np.float64) for f in init]
    for m, n in enumerate(shape):
        rest = [f for q, f in enumerate(fs) if q != m]
        kr, H = np.ones((1, R)), np.ones((R, R))
        for f in rest:
            kr, H = (kr[:, None, :] * f[None]).reshape(-1, R), H * (f.T @ f)
        fs[m] = np.linalg.solve(H, (unfold(X, m) @ kr).T).T
        bound = (bound + 1e-4) * np.linalg.cond(H)
        err = np.linalg.norm(got[off:off + n * R].reshape(n, R) - fs[m]) / np.linalg.norm(fs[m])
        assert err <= min(bound, 0.1), (m, err, bound)
        off += n * R


# leading eigenvalues 1 + delta r on both sides of the separation that the
# tridiagonalisation needs (a dozen launches; the Jacobi rotations take hundreds)
@pytest.mark.parametrize("n", [40, 160])
@pytest.mark.parametrize("delta,jacobi", [(1.2e-8, True), (5e-8, True), (2e-7, False),
                                          (1e-5, False)])
def test_svd_start_close_eigenvalues(n, delta, jacobi):
    """The eigenvectors are products of two dyadic reflections, scaled by values
    of few bits, so X is exact in FP32 and its Gram has exactly these
    eigenvalues. The result is no further from orthonormal than rounding
    exact vectors to FP32 allows: 2 |u| |2^-25 v| = 6e-8."""
    rng = np.random.default_rng(n)
    w = 1 << ((n - 1).bit_length() - 1)
    Q = np.eye(n)
    for _ in range(2):
        v = np.zeros(n)
        v[rng.permutation(n)[:w]] = 1
        v *= rng.choice([-1, 1], n)
        Q = Q @ (np.eye(n) - np.outer(v, v) * 2 / w)
    s, t = np.ones(n), np.zeros(n)
    s[9:] = np.round(np.linspace(0.95, 0.1, n - 9) * 256) / 256
    m, e = np.frexp(np.sqrt(delta * np.arange(9)[::-1]))
    t[:9] = np.ldexp(np.round(m * 1024) / 1024, e)
    X = np.concatenate([Q * s, Q * t], 1)
    assert (X.astype(np.float32) == X).all()
    ctx = tb.Context()
    before = ctx.launches
    F = tb.initialize_factors(X.reshape(n, 2, n), 8, "svd", seed=1, ctx=ctx)
    assert (ctx.launches - before > 100) == jacobi
    for V in (F[0].astype(np.float64), F[2].astype(np.float64)):
        assert np.abs(V.T @ V - np.eye(8)).max() <= 6e-8


# instances of about 100 KB, where the buffers beside them decide how many CTAs
# an SM holds: staging rows kept (few columns), given up for the second CTA
# (short rows), the second CTA given up for them (long rows)
@pytest.mark.parametrize("shape,R", [((4, 2700, 8), 4), ((4, 3200, 16), 4), ((16, 690, 48), 16),
                                     ((16, 716, 16), 16), ((9, 1450, 17), 7)])
@pytest.mark.parametrize("threads,cps", [(128, 4), (256, 2), (512, 1)])
def test_batched_large_instances(shape, R, threads, cps):
    """One sweep against FP64: row sums in FP32 to 1e-5, each solve multiplies
    the errors so far by at most the condition of its normal equations."""
    rng = np.random.default_rng(sum(shape))
    X = rng.standard_normal((3,) + shape).astype(np.float32)
    inits = [[rng.standard_normal((n, R)).astype(np.float32) for n in shape] for _ in range(3)]
    b = tb.BatchedCpAls(list(X), [R] * 3)
    b.set_config(threads, 0, cps)
    for x, init, r in zip(X, inits, b.cp_als(1, 0.0, init=inits)):
        fs, bound = [f.astype(np.float64) for f in init], 0.0
        for m, n in enumerate(shape):
            kr, H = np.ones((1, R)), np.ones((R, R))
            for q, f in enumerate(fs):
                if q != m:
                    kr, H = (kr[:, None, :] * f[None]).reshape(-1, R), H * (f.T @ f)
            fs[m] = np.linalg.solve(H, (unfold(x, m) @ kr).T).T
            bound = (bound + 1e-5) * np.linalg.cond(H)
            err = np.linalg.norm(r.factors[m] - fs[m]) / np.linalg.norm(fs[m])
            assert err <= min(bound, 0.1), (m, err, bound)
    b.close()


@pytest.mark.parametrize("shape,R,expect", [((4, 5900, 8), 4, (512, 1)),
                                            ((4, 3200, 16), 4, (256, 2)),
                                            ((16, 690, 48), 16, (512, 1)),
                                            ((20, 20, 20), 4, (256, 2))])
def test_batched_initial_config(shape, R, expect):
    """Two CTAs per SM only where the SM holds two."""
    b = tb.BatchedCpAls([np.ones(shape, np.float32)] * 400, [R] * 400)
    config = b.config
    b.close()
    assert (config["threads"], config["ctas_per_sm"]) == expect


@pytest.mark.parametrize("shape,R", [((4, 0, 3), 2), ((0, 5, 3), 2), ((4, 5, 0), 2), ((4, 5, 3), 0)])
def test_all_modes_of_an_empty_tensor(shape, R):
    """Empty sums are zero, for all modes at once as for one."""
    fs = [np.ones((n, R), np.float32) for n in shape]
    outs = tb.mttkrp_all_modes(np.ones(shape, np.float32), fs)
    for m, n in enumerate(shape):
        assert outs[m].shape == (n, R) and not outs[m].any()
        assert not tb.mttkrp(np.ones(shape, np.float32), fs, m).any()
    with pytest.raises(tb.TenrsoError, match="empty tensor"):
        tb.profile_mttkrp_dev(8, shape, [8, 8, 8], R, 0, "fp32")
