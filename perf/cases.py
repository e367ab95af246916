"""Performance cases of tenrso_b200: the calls a CP decomposition program makes.

Each case is one call (or the calls of one step) through the package's public
entry points on device-resident data, the way a program that keeps its tensor
on the GPU makes them. `kind` selects the path:

  mttkrp   mttkrp_dev for every mode of one tensor (a caller's own ALS loop)
  als      cp_als_dev, the whole decomposition from given initial factors
  als_f64  cp_als_f64 on host arrays, everything in FP64
  grad     DenseTensor.loss_grad_dev, one evaluation inside a first-order
           optimiser (the prepared tensor is kept between evaluations)
  vjp      cp_reconstruct_dev forward, reconstruction_grad_dev backward
  csf      SparseTensor.mttkrp_dev for every mode of one sparse tensor
  batched  BatchedCpAls.cp_als_dev, many small decompositions in one launch
  ttm      a chain of device n-mode products (the projection step of Tucker)
  svd      SVD-based factor initialisation on the device

Tensors are low-rank plus noise, as the decompositions meet them, or N(0,1)
where the call is linear in them; sparse indices are Zipf(1.2) per mode.
"""
import ctypes
import math
import random

import numpy as np
import torch

import tenrso_b200 as tb

DEV = "cuda"


# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest whole call: a 64^3 rank-8 decomposition, where launch
        # latency and the serial R x R steps count
        {"name": "als_64_r8_fp32", "kind": "als", "d0": 64, "d1": 64, "d2": 64, "d3": 0,
         "rank": 8, "iters": 10, "precision": "fp32", "factors": "normal", "noise": 0.01},
        # the headline decomposition: 256^3 rank 64, mixed precision
        {"name": "als_256_r64_bf16x3", "kind": "als", "d0": 256, "d1": 256, "d2": 256, "d3": 0,
         "rank": 64, "iters": 10, "precision": "bf16x3", "factors": "uniform", "noise": 0.005},
        # FP64 users: the generic element type at double, host arrays in and out
        {"name": "als_f64_120x100x80_r24", "kind": "als_f64", "d0": 120, "d1": 100, "d2": 80,
         "d3": 0, "rank": 24, "iters": 10, "factors": "normal", "noise": 0.01},
        # standalone MTTKRP, four modes, odd sizes, plain FP32
        {"name": "mttkrp_4way_odd_fp32", "kind": "mttkrp", "d0": 97, "d1": 83, "d2": 61, "d3": 45,
         "rank": 32, "precision": "fp32"},
        # standalone MTTKRP, three modes, ragged sizes, mixed precision
        {"name": "mttkrp_3way_ragged_bf16x3", "kind": "mttkrp", "d0": 301, "d1": 223, "d2": 187,
         "d3": 0, "rank": 48, "precision": "bf16x3"},
        # gradient-based fitting: loss and gradients of a 4-way tensor, FP32
        {"name": "grad_4way_r32_fp32", "kind": "grad", "d0": 128, "d1": 96, "d2": 64, "d3": 48,
         "rank": 32, "precision": "fp32"},
        # the same evaluation in mixed precision
        {"name": "grad_4way_r32_bf16x3", "kind": "grad", "d0": 128, "d1": 96, "d2": 64, "d3": 48,
         "rank": 32, "precision": "bf16x3"},
        # automatic differentiation: forward and backward of the weighted CP
        # reconstruction, odd sizes
        {"name": "vjp_4way_odd_r24", "kind": "vjp", "d0": 121, "d1": 95, "d2": 63, "d3": 47,
         "rank": 24, "precision": "fp32"},
        # sparse MTTKRP of a large recommender-like tensor
        {"name": "csf_5e7_r32", "kind": "csf", "d0": 100000, "d1": 80000, "d2": 10000,
         "nnz": 50000000, "rank": 32},
        # many small decompositions of uneven shape and rank
        {"name": "batched_512", "kind": "batched", "count": 512, "nmin": 16, "nmax": 96,
         "rmin": 4, "rmax": 16, "iters": 25, "shapes": 196},
        # Tucker projection of a cube onto three factor bases
        {"name": "ttm_256_to_64", "kind": "ttm", "d0": 256, "d1": 256, "d2": 256, "d3": 0,
         "r0": 64, "r1": 64, "r2": 64, "r3": 0},
        # the SVD start of a decomposition
        {"name": "svd_init_160x128x96_r16", "kind": "svd", "d0": 160, "d1": 128, "d2": 96,
         "d3": 0, "rank": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, ndim, lo, hi, most):
    """ndim sizes over [lo, hi], odd ones among them, with a product of at
    most `most`."""
    d = [_log_int(rng, lo, hi) for _ in range(ndim)]
    while math.prod(d) > most:
        k = max(range(ndim), key=lambda i: d[i])
        d[k] = max(2, int(d[k] * 0.9))
    return d + [0] * (4 - ndim)


def draw(rng):
    kind = rng.choice(["als", "als", "als_f64", "mttkrp", "mttkrp", "grad", "grad", "vjp", "csf",
                       "batched", "ttm", "svd"])
    case = {"kind": kind}
    if kind == "csf":
        d = [_log_int(rng, 500, 100000) for _ in range(3)]
        nnz = min(_log_int(rng, 100000, 20000000), d[0] * d[1] * d[2] // 200)
        case.update(d0=d[0], d1=d[1], d2=d[2], nnz=max(nnz, 1000), rank=rng.choice([8, 16, 32, 50]))
        return case
    if kind == "batched":
        nmin = rng.randint(8, 24)
        case.update(count=_log_int(rng, 32, 512), nmin=nmin, nmax=rng.randint(nmin + 8, 96),
                    rmin=rng.randint(2, 5), rmax=rng.randint(6, 16), iters=rng.randint(5, 25),
                    shapes=rng.randint(0, 1 << 20))
        return case
    ndim = rng.choice([3, 3, 4])
    if kind == "als":
        d = _dims(rng, ndim, 32 if ndim == 3 else 16, 256 if ndim == 3 else 96, 256 ** 3)
        case.update(rank=min(rng.choice([5, 8, 16, 24, 32, 64]), min(d[:ndim])),
                    iters=rng.randint(3, 10), precision=rng.choice(["fp32", "bf16x3"]),
                    factors="normal", noise=0.01)
    elif kind == "als_f64":
        d = _dims(rng, ndim, 24 if ndim == 3 else 12, 160 if ndim == 3 else 48, 1000000)
        case.update(rank=rng.randint(4, min(24, min(d[:ndim]))), iters=rng.randint(3, 10),
                    factors="normal", noise=0.01)
    elif kind == "mttkrp":
        d = _dims(rng, ndim, 32 if ndim == 3 else 16, 400 if ndim == 3 else 128, 30000000)
        case.update(rank=rng.choice([8, 16, 20, 32, 48, 64]),
                    precision=rng.choice(["fp32", "bf16x3"]))
    elif kind == "grad":
        d = _dims(rng, ndim, 32 if ndim == 3 else 16, 400 if ndim == 3 else 128, 37748736)
        case.update(rank=rng.choice([8, 16, 20, 32]), precision=rng.choice(["fp32", "bf16x3"]))
    elif kind == "vjp":
        d = _dims(rng, ndim, 32 if ndim == 3 else 16, 400 if ndim == 3 else 128, 37748736)
        case.update(rank=rng.choice([8, 16, 24, 32, 40]), precision="fp32")
    elif kind == "ttm":
        d = _dims(rng, ndim, 32 if ndim == 3 else 16, 400 if ndim == 3 else 96, 256 ** 3)
        for m in range(4):
            case["r%d" % m] = max(2, int(d[m] * rng.uniform(0.1, 0.4))) if m < ndim else 0
    else:
        d = _dims(rng, ndim, 24 if ndim == 3 else 12, 160 if ndim == 3 else 48, 160 * 128 * 96)
        case.update(rank=rng.randint(4, min(16, min(d[:ndim]) // 2)))
    case.update(d0=d[0], d1=d[1], d2=d[2], d3=d[3])
    return case


# ---------------------------------------------------------------------------
def _shape(case):
    return tuple(case["d%d" % m] for m in range(4) if case.get("d%d" % m, 0) > 0)


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _normal(g, *shape, dtype=torch.float32):
    return torch.randn(*shape, generator=g, device=DEV, dtype=dtype)


def _uniform(g, *shape, dtype=torch.float32):
    return torch.rand(*shape, generator=g, device=DEV, dtype=dtype)


def _kr(factors):
    """Row-wise Khatri-Rao product, the last factor's rows fastest."""
    out = factors[0]
    for f in factors[1:]:
        out = (out[:, None, :] * f[None, :, :]).reshape(-1, f.shape[1])
    return out


def _lowrank(g, shape, rank, dist, noise, scale=None):
    """Sum of `rank` rank-1 terms plus relative Gaussian noise, in FP64."""
    rnd = _normal if dist == "normal" else _uniform
    fs = [rnd(g, n, rank, dtype=torch.float64) for n in shape]
    if scale is not None:
        fs[0] = fs[0] * scale
    X = (fs[0] @ _kr(fs[1:]).T).reshape(shape)
    sigma = noise * X.norm() / math.sqrt(X.numel())
    return X + sigma * _normal(g, *shape, dtype=torch.float64)


def _dense_inputs(case, seed):
    """The case's tensor and factors (device, the case's element type)."""
    g = _gen(seed)
    shape, kind = _shape(case), case["kind"]
    if kind in ("als", "als_f64"):
        X = _lowrank(g, shape, case["rank"], case["factors"], case["noise"])
        dt = torch.float64 if kind == "als_f64" else torch.float32
        return X.to(dt), [_uniform(g, n, case["rank"], dtype=torch.float64).to(dt) for n in shape]
    if kind == "svd":
        # well separated components, as a tensor worth an SVD start has
        scale = 0.8 ** torch.arange(case["rank"], device=DEV, dtype=torch.float64)
        return _lowrank(g, shape, case["rank"], "normal", 0.01, scale).float(), []
    X = _normal(g, *shape)
    if kind == "ttm":
        return X, [_normal(g, case["r%d" % m], n) / math.sqrt(n) for m, n in enumerate(shape)]
    return X, [_normal(g, n, case["rank"]) for n in shape]


def _zipf(g, size, n):
    """n draws of a permuted Zipf(1.2) index below `size`."""
    p = torch.arange(1, size + 1, device=DEV, dtype=torch.float64) ** -1.2
    cdf = torch.cumsum(p, 0)
    z = torch.searchsorted(cdf, _uniform(g, n, dtype=torch.float64) * cdf[-1])
    perm = torch.randperm(size, generator=g, device=DEV)
    return perm[z.clamp_(max=size - 1)]


def _sparse_inputs(case, seed):
    """Distinct coordinates (nnz x 3, int64), values in (0, 1) and factors."""
    g = _gen(seed)
    shape, nnz = _shape(case), case["nnz"]
    keys = torch.empty(0, dtype=torch.int64, device=DEV)
    perms = int(torch.randint(1 << 30, (1,), generator=g, device=DEV))
    while keys.numel() < nnz:
        k = None
        for m, size in enumerate(shape):
            gm = _gen(perms + m + 7919 * keys.numel())
            i = _zipf(gm, size, 2 * nnz)
            k = i if k is None else k * size + i
        keys = torch.unique(torch.cat([keys, k]))
        del k, i
    if keys.numel() > nnz:
        keep = torch.randperm(keys.numel(), generator=g, device=DEV)[:nnz]
        keys = keys[keep.sort().values]
        del keep
    idx = torch.empty(nnz, 3, dtype=torch.int64, device=DEV)
    idx[:, 2] = keys % shape[2]
    idx[:, 1] = keys // shape[2] % shape[1]
    idx[:, 0] = keys // (shape[2] * shape[1])
    vals = 1.0 - _uniform(g, nnz)
    return idx, vals, [_uniform(g, n, case["rank"]) for n in shape]


def _batch_inputs(case, seed):
    """[(X, rank, [A, B, C])]; the shapes and ranks belong to the case."""
    g, gs = _gen(seed), random.Random(case["shapes"])
    n = case["count"]
    sizes = [[gs.randint(case["nmin"], case["nmax"]) for _ in range(3)] for _ in range(n)]
    ranks = [gs.randint(case["rmin"], min(case["rmax"], min(s))) for s in sizes]
    out = []
    for s, r in zip(sizes, ranks):
        X = _lowrank(g, s, r, "normal", 0.01).float()
        out.append((X, r, [_uniform(g, k, r) for k in s]))
    return out


def _ptrs(ts):
    return [t.data_ptr() for t in ts]


_streams = {}


def _context():
    """One context on one stream for the whole program, as a program keeps."""
    if not _streams:
        s = torch.cuda.Stream()
        _streams["s"], _streams["c"] = s, tb.Context(0, stream=s.cuda_stream)
    return _streams["c"]


class State:
    """What the program holds between calls."""

    def __init__(self, case):
        self.case = case
        self.kind = case["kind"]
        self.ctx = _context()
        self.shape = _shape(case)

    def __del__(self):
        for name in ("dense", "sparse", "batch"):
            if getattr(self, name, None) is not None:
                getattr(self, name).close()


def prepare(case, seed):
    st = State(case)
    if st.kind == "csf":
        idx, vals, st.factors = _sparse_inputs(case, seed)
        torch.cuda.synchronize()
        st.sparse = tb.SparseTensor(ctx=st.ctx, d_indices=idx.data_ptr(),
                                    d_values=vals.data_ptr(), nnz=case["nnz"], shape=st.shape)
        st.out = [torch.empty(n, case["rank"], device=DEV) for n in st.shape]
        return st
    if st.kind == "batched":
        items = _batch_inputs(case, seed)
        st.batch = tb.BatchedCpAls([X.cpu().numpy() for X, _, _ in items],
                                   [r for _, r, _ in items], ctx=st.ctx)
        st.init = torch.from_numpy(st.batch.pack([[f.cpu().numpy() for f in fs]
                                                  for _, _, fs in items])).cuda()
        st.out = torch.empty_like(st.init)
        torch.cuda.synchronize()
        return st
    st.X, st.factors = _dense_inputs(case, seed)
    if st.kind == "als_f64":
        st.X = st.X.cpu().numpy()
        st.factors = [f.cpu().numpy() for f in st.factors]
        return st
    if st.kind == "als":
        st.init = torch.cat([f.reshape(-1) for f in st.factors])
        st.out = torch.empty_like(st.init)
    elif st.kind == "grad":
        torch.cuda.synchronize()
        st.dense = tb.DenseTensor(st.X.data_ptr(), st.shape, case["precision"], ctx=st.ctx)
        st.out = [torch.empty_like(f) for f in st.factors]
    elif st.kind == "vjp":
        st.weights = _uniform(_gen(seed + 1000003), case["rank"]) + 0.5
        st.forward = torch.empty(st.shape, device=DEV)
        st.out = [torch.empty_like(f) for f in st.factors]
    elif st.kind == "ttm":
        cur, st.out = list(st.shape), []
        for m, f in enumerate(st.factors):
            cur[m] = f.shape[0]
            st.out.append(torch.empty(cur, device=DEV))
    elif st.kind == "svd":
        st.out = torch.empty(sum(st.shape) * case["rank"], device=DEV)
    else:
        st.out = [torch.empty_like(f) for f in st.factors]
    torch.cuda.synchronize()
    return st


def _i64(shape):
    return (ctypes.c_int64 * len(shape))(*shape)


def run(st):
    case, shape = st.case, st.shape
    if st.kind == "als":
        fit, _, _ = tb.cp_als_dev(st.X.data_ptr(), shape, case["rank"], case["iters"], 0.0,
                                  st.init.data_ptr(), st.out.data_ptr(), case["precision"],
                                  ctx=st.ctx)
        return {"factors": st.out, "fit": fit}
    if st.kind == "als_f64":
        d = tb.cp_als_f64(st.X, case["rank"], case["iters"], 0.0, init=st.factors, ctx=st.ctx)
        return {"factors": np.concatenate([f.reshape(-1) for f in d.factors]), "fit": d.fit}
    if st.kind == "mttkrp":
        for m in range(len(shape)):
            tb.mttkrp_dev(st.X.data_ptr(), shape, _ptrs(st.factors), case["rank"], m,
                          st.out[m].data_ptr(), case["precision"], ctx=st.ctx)
        return st.out
    if st.kind == "grad":
        loss = st.dense.loss_grad_dev(_ptrs(st.factors), case["rank"], 1e-3, _ptrs(st.out))
        return {"grads": st.out, "loss": loss}
    if st.kind == "vjp":
        tb.cp_reconstruct_dev(_ptrs(st.factors), shape, case["rank"], st.forward.data_ptr(),
                              st.weights.data_ptr(), ctx=st.ctx)
        tb.reconstruction_grad_dev(st.X.data_ptr(), shape, _ptrs(st.factors), case["rank"],
                                   _ptrs(st.out), st.weights.data_ptr(), case["precision"],
                                   ctx=st.ctx)
        return {"forward": st.forward, "grads": st.out}
    if st.kind == "csf":
        for m in range(3):
            st.sparse.mttkrp_dev(_ptrs(st.factors), case["rank"], m, st.out[m].data_ptr())
        return st.out
    if st.kind == "batched":
        st.batch.cp_als_dev(case["iters"], 0.0, st.init.data_ptr(), st.out.data_ptr())
        return st.out
    lib = tb.load()
    if st.kind == "ttm":
        cur, src = list(shape), st.X
        for m, f in enumerate(st.factors):
            rc = lib.tsr_nmode_product_dev_f32(st.ctx.handle, src.data_ptr(), len(cur), _i64(cur),
                                               f.data_ptr(), f.shape[0], f.shape[1], m,
                                               st.out[m].data_ptr())
            if rc:
                raise tb.TenrsoError(rc, lib.tsr_last_error().decode())
            cur[m], src = f.shape[0], st.out[m]
        return src
    rc = lib.tsr_cp_init_dev_f32(st.ctx.handle, st.X.data_ptr(), len(shape), _i64(shape),
                                 case["rank"], 2, 0, st.out.data_ptr())
    if rc:
        raise tb.TenrsoError(rc, lib.tsr_last_error().decode())
    return st.out


# ---------------------------------------------------------------------------
def work(case):
    """Bytes and operations of one pass. An ALS iteration needs each mode's
    MTTKRP (2 |X| R operations each) but can keep X on the chip only when it
    fits, so X counts once per call; factors are read and written once."""
    shape, kind, R = _shape(case), case["kind"], case.get("rank", 0)
    n, nd = math.prod(shape) if shape else 0, len(shape)
    fl = sum(shape) * R
    if kind == "als":
        return {"bytes": 4 * (n + 2 * fl), "flops": 2 * n * R * nd * case["iters"]}
    if kind == "als_f64":
        return {"bytes": 8 * (n + 2 * fl), "flops": 2 * n * R * nd * case["iters"]}
    if kind in ("mttkrp", "grad"):
        return {"bytes": 4 * (n + 2 * fl), "flops": 2 * n * R * nd}
    if kind == "vjp":
        return {"bytes": 4 * (2 * n + 2 * fl), "flops": 2 * n * R * (nd + 1)}
    if kind == "csf":
        return {"bytes": 16 * case["nnz"] + 8 * fl, "flops": 3 * 3 * case["nnz"] * R}
    if kind == "batched":
        n = case["count"] * ((case["nmin"] + case["nmax"]) / 2) ** 3
        r = (case["rmin"] + case["rmax"]) / 2
        return {"bytes": 4 * n, "flops": 2 * n * r * 3 * case["iters"]}
    if kind == "ttm":
        cur, flops = list(shape), 0
        for m in range(nd):
            flops += 2 * math.prod(cur) * case["r%d" % m]
            cur[m] = case["r%d" % m]
        return {"bytes": 4 * (n + math.prod(cur)), "flops": flops}
    return {"bytes": 4 * (n + fl), "flops": sum(n * s + 9 * s ** 3 for s in shape)}


# ---------------------------------------------------------------------------
def _mttkrp64(X, factors, mode):
    """MTTKRP of one mode in FP64; the tensor's leading mode stays outermost."""
    Xn = X.movedim(mode, 0).reshape(X.shape[mode], -1)
    return Xn @ _kr([f for m, f in enumerate(factors) if m != mode])


def _had(grams, skip=None):
    out = None
    for m, G in enumerate(grams):
        if m != skip:
            out = G.clone() if out is None else out * G
    return out


def _als64(X, factors, iters):
    """cp_als in FP64: (factors, fit)."""
    fs = [f.clone() for f in factors]
    grams = [f.T @ f for f in fs]
    nx2 = (X * X).sum()
    fit = 0.0
    for _ in range(iters):
        for m in range(X.dim()):
            M = _mttkrp64(X, fs, m)
            fs[m] = torch.linalg.solve(_had(grams, m), M.T).T.contiguous()
            grams[m] = fs[m].T @ fs[m]
        err2 = nx2 - 2 * (M * fs[-1]).sum() + _had(grams).sum()
        fit = 1.0 - math.sqrt(max(float(err2 / nx2), 0.0))
    return fs, min(max(fit, 0.0), 1.0)


def _exact_batched(items, iters):
    """All instances at once, zero-padded to the largest shape and rank; the
    padded columns get a unit diagonal in the normal equations."""
    out = []
    for lo in range(0, len(items), 64):
        part = items[lo:lo + 64]
        R = max(r for _, r, _ in part)
        S = [max(X.shape[m] for X, _, _ in part) for m in range(3)]
        X = torch.zeros(len(part), *S, device=DEV, dtype=torch.float64)
        F = [torch.zeros(len(part), S[m], R, device=DEV, dtype=torch.float64) for m in range(3)]
        one = torch.zeros(len(part), R, device=DEV, dtype=torch.float64)
        for b, (x, r, fs) in enumerate(part):
            X[b, :x.shape[0], :x.shape[1], :x.shape[2]] = x
            one[b, r:] = 1.0
            for m in range(3):
                F[m][b, :x.shape[m], :r] = fs[m]
        eye = torch.diag_embed(one)
        for _ in range(iters):
            for m in range(3):
                a, c = [q for q in range(3) if q != m]
                kr = (F[a][:, :, None, :] * F[c][:, None, :, :]).reshape(len(part), -1, R)
                M = X.movedim(m + 1, 1).reshape(len(part), S[m], -1) @ kr
                G = (F[a].transpose(1, 2) @ F[a]) * (F[c].transpose(1, 2) @ F[c]) + eye
                F[m] = torch.linalg.solve(G, M.transpose(1, 2)).transpose(1, 2).contiguous()
        for b, (x, r, _) in enumerate(part):
            out += [F[m][b, :x.shape[m], :r].reshape(-1) for m in range(3)]
    return torch.cat(out)


def exact(case, seed):
    kind = case["kind"]
    if kind == "csf":
        idx, vals, fs = _sparse_inputs(case, seed)
        vals, fs = vals.double(), [f.double() for f in fs]
        outs = [torch.zeros_like(f) for f in fs]
        for lo in range(0, case["nnz"], 2000000):
            i, v = idx[lo:lo + 2000000], vals[lo:lo + 2000000, None]
            rows = [f[i[:, m]] for m, f in enumerate(fs)]
            for m in range(3):
                a, b = [q for q in range(3) if q != m]
                outs[m].index_add_(0, i[:, m], v * rows[a] * rows[b])
        return outs
    if kind == "batched":
        items = _batch_inputs(case, seed)
        return _exact_batched([(X.double(), r, [f.double() for f in fs]) for X, r, fs in items],
                              case["iters"])
    X, fs = _dense_inputs(case, seed)
    X, fs = X.double(), [f.double() for f in fs]
    if kind in ("als", "als_f64"):
        fs, fit = _als64(X, fs, case["iters"])
        return {"factors": torch.cat([f.reshape(-1) for f in fs]), "fit": fit}
    if kind == "mttkrp":
        return [_mttkrp64(X, fs, m) for m in range(X.dim())]
    if kind == "grad":
        E = (fs[0] @ _kr(fs[1:]).T).reshape(X.shape) - X
        grads = [2 * _mttkrp64(E, fs, m) + 2e-3 * fs[m] for m in range(X.dim())]
        return {"grads": grads, "loss": float((E * E).sum()) + 1e-3 * sum(float((f * f).sum())
                                                                         for f in fs)}
    if kind == "vjp":
        w = (_uniform(_gen(seed + 1000003), case["rank"]) + 0.5).double()
        return {"forward": ((fs[0] * w) @ _kr(fs[1:]).T).reshape(X.shape),
                "grads": [_mttkrp64(X, fs, m) * w for m in range(X.dim())]}
    if kind == "ttm":
        for m, f in enumerate(fs):
            X = torch.tensordot(f, X, dims=([1], [m])).movedim(0, m)
        return X
    out = []
    for m in range(X.dim()):
        Xn = X.movedim(m, 0).reshape(X.shape[m], -1)
        lam, V = torch.linalg.eigh(Xn @ Xn.T)
        u = V.flip(1)[:, :case["rank"]]
        top = u.gather(0, u.abs().argmax(0, keepdim=True))
        out.append((u * top.sign()).reshape(-1))
    return torch.cat(out)
