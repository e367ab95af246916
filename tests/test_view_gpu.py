"""The kernels that read a row-major tensor in place: MTTKRP in FP32 and FP64,
n-mode products, the two-pass reconstruction gradient, and the FP32 route of
BF16x3 requests, at the sizes where their tiles, runs and load patterns change.

Tolerances against FP64, relative Frobenius: FP32 sums of N(0,1) products, in
chains of 16 columns or of at most 130 terms, 1e-5 (the bound of the other FP32
MTTKRP tests); BF16x3 1e-4; FP64 1e-12; reconstruction, at most 66 products per
entry, 1e-6."""
import ctypes as C

import numpy as np
import pytest

import tenrso_b200 as tb
from tenrso_b200 import _lib

pytestmark = pytest.mark.gpu


def rel(a, b):
    b = np.asarray(b, np.float64)
    return np.linalg.norm(np.asarray(a, np.float64) - b) / max(np.linalg.norm(b), 1e-300)


def mttkrp64(X, fs, mode):
    kr = np.ones((1, fs[0].shape[1]))
    for m, f in enumerate(fs):
        if m != mode:
            kr = (kr[:, None, :] * f.astype(np.float64)[None]).reshape(-1, kr.shape[1])
    return np.moveaxis(X.astype(np.float64), mode, 0).reshape(X.shape[mode], -1) @ kr


def device(a, offset=0):
    """A copy of `a` on the GPU that starts `offset` elements into its buffer."""
    import torch
    buf = torch.empty(a.size + offset, dtype=torch.float32, device="cuda")
    t = buf[offset:].reshape(a.shape)
    t.copy_(torch.from_numpy(a))
    return t


def draw(shape, R, seed=7):
    rng = np.random.default_rng(seed)
    return (rng.standard_normal(shape).astype(np.float32),
            [rng.standard_normal((n, R)).astype(np.float32) for n in shape])


# rows across every tile height (32..128) and remainder, runs of 1 to 300
# columns, inner modes too short to be the run, ranks across the column tiles
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("shape,R", [
    ((131, 7, 259), 33), ((64, 1, 64), 8), ((1, 1, 1), 1), ((16, 16, 16), 65), ((33, 48, 2), 16),
    ((97, 129), 100), ((5, 300, 3), 24), ((65, 3, 2, 130), 17), ((2, 3, 4, 5, 6, 7), 9),
    ((1000, 4, 3), 48), ((12, 20, 31, 8), 130)])
def test_mttkrp_fp32(shape, R, offset):
    import torch
    X, fs = draw(shape, R)
    ctx = tb.Context()
    dX, dfs = device(X, offset), [device(f, offset) for f in fs]
    for mode in range(len(shape)):
        out = torch.empty(shape[mode], R, device="cuda")
        torch.cuda.synchronize()
        tb.mttkrp_dev(dX.data_ptr(), shape, [f.data_ptr() for f in dfs], R, mode, out.data_ptr(),
                      "fp32", ctx=ctx)
        ctx.synchronize()
        assert rel(out.cpu().numpy(), mttkrp64(X, fs, mode)) <= 1e-5, mode


def test_mttkrp_fp32_nonfinite_rows():
    """A NaN or infinity reaches its own output row and no other."""
    X, fs = draw((40, 37, 29), 20)
    X[3, 5, 7], X[11, 13, 17] = np.nan, np.inf
    for mode in range(3):
        bad = np.zeros(X.shape[mode], bool)
        bad[[(3, 5, 7)[mode], (11, 13, 17)[mode]]] = True
        got = tb.mttkrp(X, fs, mode, precision="fp32")
        assert not np.isfinite(got[bad]).any() and np.isfinite(got[~bad]).all()
        ok = mttkrp64(np.where(np.isfinite(X), X, 0), fs, mode)
        assert rel(got[~bad], ok[~bad]) <= 1e-5


# both sides of the rank where a single BF16x3 call stops running in FP32,
# three modes with odd sizes, four modes with runs that suit the tensor-core
# kernel and with short ones, and two modes
@pytest.mark.parametrize("shape", [(61, 43, 27), (20, 24, 16, 64), (19, 13, 11, 9), (70, 45)])
@pytest.mark.parametrize("R", [5, 48, 49, 128, 129])
def test_bf16x3_route(shape, R):
    X, fs = draw(shape, R)
    for mode in range(len(shape)):
        got = tb.mttkrp(X, fs, mode, precision="bf16x3")
        assert rel(got, mttkrp64(X, fs, mode)) <= 1e-4, mode


@pytest.mark.parametrize("shape,R", [((129, 5, 67), 25), ((3, 4, 300), 65), ((17, 2, 9, 33), 8),
                                     ((200, 130), 24), ((1, 7, 1), 3)])
def test_mttkrp_f64(shape, R):
    rng = np.random.default_rng(3)
    X = rng.standard_normal(shape)
    fs = [rng.standard_normal((n, R)) for n in shape]
    for mode in range(len(shape)):
        assert rel(tb.mttkrp_f64(X, fs, mode), mttkrp64(X, fs, mode)) <= 1e-12, mode


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("shape,J", [((130, 66, 33), 65), ((4, 128, 64), 64), ((7, 31, 1), 130),
                                     ((1, 33, 257), 3), ((70000, 2, 3), 2)])
def test_matrix_product(shape, J, offset):
    import torch
    rng = np.random.default_rng(J)
    X = rng.standard_normal(shape).astype(np.float32)
    ctx, lib = tb.Context(), _lib.load()
    dX = device(X, offset)
    for mode in range(3):
        M = rng.standard_normal((J, shape[mode])).astype(np.float32)
        dM = device(M, offset)
        oshape = shape[:mode] + (J,) + shape[mode + 1:]
        out = torch.empty(oshape, device="cuda")
        torch.cuda.synchronize()
        rc = lib.tsr_nmode_product_dev_f32(ctx.handle, dX.data_ptr(), 3, (C.c_int64 * 3)(*shape),
                                           dM.data_ptr(), J, shape[mode], mode, out.data_ptr())
        assert rc == 0
        ctx.synchronize()
        ref = np.moveaxis(np.tensordot(M.astype(np.float64), X, (1, mode)), 0, mode)
        assert rel(out.cpu().numpy(), ref) <= 1e-5, mode


# two passes (both sides at least R wide) and one pass per mode (the others)
@pytest.mark.parametrize("shape,R", [((65, 7, 33), 24), ((9, 8, 7, 6), 33), ((3, 4, 2, 5, 3), 6),
                                     ((4, 30, 20), 5), ((130, 3, 2), 7), ((40, 50), 8)])
@pytest.mark.parametrize("precision", ["fp32", "bf16x3"])
def test_reconstruction_grad(shape, R, precision):
    import torch
    G, fs = draw(shape, R)
    w = np.random.default_rng(1).random(R).astype(np.float32) + 0.5
    ctx = tb.Context()
    dG, dw, dfs = device(G, 1), device(w), [device(f) for f in fs]
    outs = [torch.empty_like(f) for f in dfs]
    torch.cuda.synchronize()
    tb.reconstruction_grad_dev(dG.data_ptr(), shape, [f.data_ptr() for f in dfs], R,
                               [o.data_ptr() for o in outs], dw.data_ptr(), precision, ctx=ctx)
    ctx.synchronize()
    for mode, o in enumerate(outs):
        bound = 1e-5 if precision == "fp32" else 1e-4
        assert rel(o.cpu().numpy(), mttkrp64(G, fs, mode) * w) <= bound, mode


@pytest.mark.parametrize("shape,R", [((129, 3, 43), 33), ((128, 128), 32), ((257, 1, 2), 66),
                                     ((1, 127, 3), 1), ((5, 26, 4, 65), 24)])
def test_reconstruct_tiles(shape, R):
    _, fs = draw(shape, R)
    ref = (fs[0].astype(np.float64) @ _kr(fs[1:]).T).reshape(shape)
    assert rel(tb.cp_reconstruct(fs), ref) <= 1e-6


def _kr(fs):
    out = fs[0].astype(np.float64)
    for f in fs[1:]:
        out = (out[:, None, :] * f[None]).reshape(-1, out.shape[1])
    return out


# both sides of the rule: a short mode beside a long one leaves the contraction
# of the two passes few blocks of many steps, so those run one pass (two
# launches) per mode; the others at most five launches in all
@pytest.mark.parametrize("shape,R,per_mode", [((60, 2, 3000), 16, True),
                                              ((60, 3000, 2), 16, True),
                                              ((6, 1200, 2, 2, 6), 16, True),
                                              ((60, 2, 300), 16, False),
                                              ((64, 30, 47), 24, False),
                                              ((6, 12, 2, 2, 16), 16, False)])
@pytest.mark.parametrize("precision", ["fp32", "bf16x3"])
def test_reconstruction_grad_route(shape, R, per_mode, precision):
    import torch
    G, fs = draw(shape, R)
    ctx = tb.Context()
    dG, dfs = device(G), [device(f) for f in fs]
    outs = [torch.empty_like(f) for f in dfs]
    torch.cuda.synchronize()
    before = ctx.launches
    tb.reconstruction_grad_dev(dG.data_ptr(), shape, [f.data_ptr() for f in dfs], R,
                               [o.data_ptr() for o in outs], None, precision, ctx=ctx)
    ctx.synchronize()
    launches = ctx.launches - before
    assert launches == 2 * len(shape) if per_mode else launches <= 5
    for mode, o in enumerate(outs):
        assert rel(o.cpu().numpy(), mttkrp64(G, fs, mode)) <= 1e-5, mode


# a prepared BF16x3 tensor whose view suits no copy: two FP32 passes (at most
# six launches) where they pay, else one tensor-core pass and one gradient
# kernel per mode
@pytest.mark.parametrize("shape,R,per_mode", [((11, 21, 4001), 32, True), ((5, 9, 4001), 32, True),
                                              ((61, 43, 27), 16, False),
                                              ((19, 13, 11, 9), 8, False)])
def test_loss_grad_route(shape, R, per_mode):
    import torch
    X, fs = draw(shape, R)
    ctx = tb.Context()
    dX, dfs = device(X), [device(f) for f in fs]
    outs = [torch.empty_like(f) for f in dfs]
    torch.cuda.synchronize()
    D = tb.DenseTensor(dX.data_ptr(), shape, "bf16x3", ctx=ctx)
    before = ctx.launches
    loss = D.loss_grad_dev([f.data_ptr() for f in dfs], R, 1e-3, [o.data_ptr() for o in outs])
    launches = ctx.launches - before
    D.close()
    assert launches >= 2 + 2 * len(shape) if per_mode else launches <= 6
    f64 = [f.astype(np.float64) for f in fs]
    E = (f64[0] @ _kr(fs[1:]).T).reshape(shape) - X
    assert abs(loss - (E ** 2).sum() - 1e-3 * sum((f ** 2).sum() for f in f64)) <= 1e-4 * loss
    for mode, o in enumerate(outs):
        ref = 2 * np.moveaxis(E, mode, 0).reshape(shape[mode], -1) @ _kr(
            [f for m, f in enumerate(fs) if m != mode]) + 2e-3 * f64[mode]
        assert rel(o.cpu().numpy(), ref) <= 1e-4, mode


# where a single BF16x3 call writes a bf16 unfolding and runs the tensor cores
# (three launches), and where it reads X in FP32 (two): ranks, modes, column
# counts and tensor sizes on both sides of the rule
@pytest.mark.parametrize("shape,R,tensor_cores", [
    ((258, 260, 252), 36, {0}), ((258, 260, 252), 64, {0}), ((258, 260, 252), 116, {0}),
    ((258, 260, 252), 32, set()), ((258, 260, 252), 50, set()), ((258, 260, 252), 96, set()),
    ((250, 260, 252), 64, set()), ((261, 259, 251), 64, set()), ((65, 64, 66, 64), 48, {1}),
    ((65, 64, 66, 64), 68, set()), ((65, 64, 66, 63), 48, set()), ((4100, 4100), 64, {0})])
def test_bf16x3_large_route(shape, R, tensor_cores):
    import torch
    g = torch.Generator(device="cuda").manual_seed(5)
    X = torch.randn(*shape, generator=g, device="cuda")
    fs = [torch.randn(n, R, generator=g, device="cuda") for n in shape]
    ctx = tb.Context()
    for mode in range(len(shape)):
        out = torch.empty(shape[mode], R, device="cuda")
        torch.cuda.synchronize()
        before = ctx.launches
        tb.mttkrp_dev(X.data_ptr(), shape, [f.data_ptr() for f in fs], R, mode, out.data_ptr(),
                      "bf16x3", ctx=ctx)
        assert ctx.launches - before == (3 if mode in tensor_cores else 2), mode
        kr = torch.ones(1, R, device="cuda", dtype=torch.float64)
        for m, f in enumerate(fs):
            if m != mode:
                kr = (kr[:, None, :] * f.double()[None]).reshape(-1, R)
        ref = X.double().movedim(mode, 0).reshape(shape[mode], -1) @ kr
        bound = 1e-4 if mode in tensor_cores else 1e-5
        assert float((out.double() - ref).norm() / ref.norm()) <= bound, mode


# more column tiles than one launch holds, in both output layouts; contractions
# shorter than a chunk, expanding, with rows on both sides of a tile
@pytest.mark.parametrize("A,I,B,J", [(1, 2, 3, 65535 * 32 + 17), (2, 2, 1, 65535 * 16 + 17),
                                     (1, 16, 3001, 64), (301, 5, 5, 301), (3, 1, 130, 33),
                                     (2, 30, 127, 48), (40, 10, 10, 65)])
def test_matrix_product_expanding(A, I, B, J):
    """At most 30 products per entry: the reconstruction's bound."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(J)
    X = torch.randn(A, I, B, generator=g, device="cuda")
    M = torch.randn(J, I, generator=g, device="cuda")
    out = torch.empty(A, J, B, device="cuda")
    torch.cuda.synchronize()
    ctx, lib = tb.Context(), _lib.load()
    assert lib.tsr_nmode_product_dev_f32(ctx.handle, X.data_ptr(), 3, (C.c_int64 * 3)(A, I, B),
                                         M.data_ptr(), J, I, 1, out.data_ptr()) == 0
    ctx.synchronize()
    ref = torch.einsum("ji,aib->ajb", M.double(), X.double())
    assert float((out.double() - ref).norm() / ref.norm()) <= 1e-6


@pytest.mark.parametrize("shape,R", [((97, 83, 61, 45), 32), ((301, 223, 187), 48),
                                     ((3000, 2500), 20)])
def test_mttkrp_fp32_chains(shape, R):
    """The error of sums in chains of 16 columns, collected once more per split.
    With u = 2^-24, N(0,1) terms and splits of n chains, the relative error is
    about u sqrt(2.8 + n / 6): the rounding of a partial sum of j terms has the
    variance j u^2 / 3. Splits have at most 60 chains here: 2.2e-7 at most, half
    as much again allowed. One chain per split would give up to 7e-7."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(11)
    X = torch.randn(*shape, generator=g, device="cuda")
    fs = [torch.randn(n, R, generator=g, device="cuda") for n in shape]
    ctx = tb.Context()
    for mode in range(len(shape)):
        out = torch.empty(shape[mode], R, device="cuda")
        torch.cuda.synchronize()
        tb.mttkrp_dev(X.data_ptr(), shape, [f.data_ptr() for f in fs], R, mode, out.data_ptr(),
                      "fp32", ctx=ctx)
        kr = torch.ones(1, R, device="cuda", dtype=torch.float64)
        for m, f in enumerate(fs):
            if m != mode:
                kr = (kr[:, None, :] * f.double()[None]).reshape(-1, R)
        ref = X.double().movedim(mode, 0).reshape(shape[mode], -1) @ kr
        assert float((out.double() - ref).norm() / ref.norm()) <= 3.3e-7, mode
