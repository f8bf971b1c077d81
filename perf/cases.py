"""Performance cases: what programs that use this library have it do.

Most programs keep a matrix on the GPU and multiply with it many times
(``sbb.device.Plan``); some multiply once with each new matrix (``csr5_kernel``
on device pointers, a plan with the learned kernel choice); some hand over host
arrays, as the drop-in entry points take them; some run many matrices of
uneven sizes as one batch; and the kernel selector is trained on the GPU.  The
matrices are the seeded families of ``sbb.gen`` with the sizes of the benchmark
and test configurations, made here on the GPU with torch.

A case is a dict of plain values:

  op      "spmv"   one y = alpha*A*x + beta*y with a plan that is kept
          "once"   a matrix used once: plan, product, release
          "batch"  every product of a batch, replayed from its CUDA graph
          "host"   one host-pointer entry point, arrays in pinned memory
          "train"  full-batch training of the selector's network
  family, m, n and the family's parameters: the matrix (see ``_matrix``)
  kernel, form, alpha, beta and the entry point's other arguments

``work`` counts the bytes that y = alpha*A*x + beta*y cannot do without: 12 per
nnz (FP32 storage: 8), the row pointer, x, y written, and y read when beta is
not zero.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(1, os.path.abspath("sparse-blas_b200"))

import sbb  # noqa: E402
from sbb import api, gen, selector  # noqa: E402
from sbb.batch import Batch  # noqa: E402
from sbb.device import Plan  # noqa: E402

# ---- the cases -------------------------------------------------------------


def listed():
    return [
        # A small solver's product: 10,000 power-law rows, everything in L2;
        # launches and the host's share of the call count.
        dict(name="spmv_powerlaw_10k", op="spmv", family="powerlaw", m=10_000, n=10_000, expo=2.0,
             lmin=1.0, lmax=1000.0, kernel="auto", form="f64", alpha=1.0, beta=0.0),
        # A stencil-like matrix: short, even rows near the diagonal, an odd
        # number of them (the automatic choice takes the vector kernel).
        dict(name="spmv_banded_200k", op="spmv", family="banded", m=199_999, n=199_999, hw=32,
             r=24.0, kernel="auto", form="f64", alpha=1.0, beta=0.5),
        # A rail-scheduling-like constraint matrix: few, long, uneven rows
        # over a wide x, all values one.
        dict(name="spmv_shortwide_4284", op="spmv", family="shortwide", m=4284, n=1_092_610,
             mean=2640.0, sigma=1.0, kernel="auto", form="f64", alpha=1.0, beta=0.0),
        # The headline product: a circuit matrix, 60M nnz, a few dense rows.
        dict(name="spmv_circuit_5.5M", op="spmv", family="circuit", m=5_500_000, n=5_500_000,
             kernel="auto", form="f64", alpha=1.0, beta=0.5),
        # The same product with values and x stored in FP32.
        dict(name="spmv_circuit_5.5M_f32", op="spmv", family="circuit", m=5_500_000, n=5_500_000,
             kernel="auto", form="f32", alpha=1.0, beta=0.5),
        # FP32 storage with FP32 lane sums on dense diagonal blocks.
        dict(name="spmv_blocks_150k_lanes", op="spmv", family="blockdiag", m=150_001, n=150_001,
             block=256, r=100.0, kernel="auto", form="lanes", alpha=1.0, beta=0.0),
        # The merge-path kernel (kernel 2 of the drop-in entry points) as a
        # kept plan on a circuit matrix of ordinary size.
        dict(name="spmv_circuit_700k_merge", op="spmv", family="circuit", m=700_001, n=700_001,
             kernel="merge", form="f64", alpha=-0.7, beta=0.3),
        # Many systems at once: 512 matrices of 1k to 200k rows, classes by
        # the trained selector, one CUDA graph.
        dict(name="batch_512", op="batch", count=512, base=5, nmin=1_000, nmax=200_000, beta=0.5),
        # A matrix that is used once, on device pointers, by the reference's
        # csr5_kernel entry point (which builds its tiles in every call).
        dict(name="once_csr5_circuit_1.4M", op="once", entry="csr5", family="circuit",
             m=1_375_000, n=1_375_000, alpha=1.0, beta=0.0),
        # A new matrix whose kernel the trained network picks.
        dict(name="once_learned_30k", op="once", entry="learned", family="plfamily", m=30_011,
             n=30_011, expo=2.5, r=20.0, alpha=1.0, beta=0.5),
        # A caller with host arrays: spMV_mgpu_v1, kernel 2.
        dict(name="host_v1_circuit_100k", op="host", entry="v1", kernel=2, family="circuit",
             m=100_003, n=100_003, alpha=1.0, beta=0.5),
        # Training the selector: 4,000 timed matrices, forward and backward
        # pass and Adam, the first 50 of the steps that a training takes.
        dict(name="train_selector_4000", op="train", samples=4000, steps=50),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_matrix(rng, families, mmax, nnzmax):
    f = rng.choice(families)
    scal = dict(alpha=rng.choice([1.0, 1.0, -0.7]), beta=rng.choice([0.0, 0.5, 0.3]))
    if f == "circuit":
        m = _logint(rng, min(20_000, mmax // 4), mmax)
        return dict(family=f, m=m, n=m, **scal)
    if f == "shortwide":
        m, mean = _logint(rng, 500, 20_000), float(_logint(rng, 300, 3000))
        return dict(family=f, m=m, n=_logint(rng, 200_000, 2_000_000), mean=mean, sigma=1.0, **scal)
    if f == "powerlaw":
        m = _logint(rng, 1000, min(mmax, 1_000_000))
        return dict(family=f, m=m, n=m, expo=2.0, lmin=1.0, lmax=1000.0, **scal)
    if f == "uniform":  # rectangular, short rows, some of them empty
        return dict(family=f, m=_logint(rng, 1000, min(mmax, 2_000_000)),
                    n=_logint(rng, 1000, 2_000_000), lmax=rng.choice([4, 8, 30]),
                    p_empty=rng.choice([0.0, 0.1, 0.5]), **scal)
    m = _logint(rng, 1000, min(mmax, 1_000_000))
    r = float(min(_logint(rng, 4, 200), max(4, nnzmax // m)))
    if f == "banded":
        return dict(family=f, m=m, n=m, hw=rng.randint(1, 64), r=r, **scal)
    if f == "blockdiag":
        return dict(family=f, m=m, n=m, block=rng.randint(16, 256), r=r, **scal)
    return dict(family="plfamily", m=m, n=m, expo=rng.uniform(1.6, 3.0), r=r, **scal)


EVERY = ["powerlaw", "banded", "blockdiag", "plfamily", "circuit", "shortwide", "uniform"]


def draw(rng):
    op = rng.choices(["spmv", "once", "batch", "host", "train"], [50, 16, 12, 14, 8])[0]
    if op == "spmv":
        c = _draw_matrix(rng, EVERY, 5_500_000, 40_000_000)
        form = rng.choices(["f64", "f32", "lanes"], [60, 25, 15])[0]
        kernel = "auto" if form == "lanes" else rng.choices(
            ["auto", "merge", "tiled", "learned"], [60, 15, 15, 10])[0]
        if c["family"] in ("banded", "blockdiag") and form != "lanes" and rng.random() < 0.2:
            kernel = "vector"
        return dict(op=op, kernel=kernel, form=form, **c)
    if op == "once":
        return dict(op=op, entry=rng.choice(["csr5", "learned"]),
                    **_draw_matrix(rng, EVERY, 3_000_000, 20_000_000))
    if op == "batch":
        lo = _logint(rng, 500, 4000)
        return dict(op=op, count=_logint(rng, 8, 160), base=rng.randint(1000, 9000), nmin=lo,
                    nmax=lo * rng.randint(10, 40), beta=rng.choice([0.0, 0.5]))
    if op == "host":
        c = _draw_matrix(rng, ["powerlaw", "banded", "plfamily", "circuit", "uniform"], 800_000,
                         8_000_000)
        entry = rng.choice(["baseline", "v1", "v2"])
        return dict(op=op, entry=entry, kernel=rng.choice([1, 2, 3]), tasks=8, q=2, **c)
    return dict(op=op, samples=_logint(rng, 250, 4000), steps=rng.randint(10, 50))


# ---- matrices --------------------------------------------------------------


def _powerlaw(u, e, a, b):
    """Truncated power law, density ~ x^-e on [a, b], from uniform u."""
    if abs(e - 1.0) < 1e-12:
        return a * (b / a) ** u
    k = 1.0 - e
    return (a ** k + u * (b ** k - a ** k)) ** (1.0 / k)


class _Rand:
    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)

    def uni(self, *shape):
        return torch.rand(shape, generator=self.g, device="cuda", dtype=torch.float64)

    def below(self, limit, count):
        return (self.uni(count) * limit).long().clamp_(max=limit - 1)

    def sym(self, count):
        return self.uni(count).mul_(2.0).sub_(1.0)


def _window(R, m, n, lo, w, r):
    """Row i: round(r*U(0.5, 1.5)) distinct columns of [lo_i, lo_i + w_i)."""
    L = torch.minimum((r * (0.5 + R.uni(m))).round().long().clamp_(min=1), w)
    W = int(w.max())
    keys = []
    step = max(1, 16_000_000 // W)
    slot = torch.arange(W, device="cuda")
    for a in range(0, m, step):
        b = min(m, a + step)
        u = torch.rand(b - a, W, generator=R.g, device="cuda")
        u.masked_fill_(slot[None, :] >= w[a:b, None], 2.0)
        nth = u.sort(dim=1).values.gather(1, L[a:b, None] - 1)
        rows, cols = (u <= nth).nonzero(as_tuple=True)
        keys.append((rows + a) * n + cols + lo[rows + a])
    return torch.cat(keys)


def _keys(c, R):
    """Sorted row*n + column of every nnz of the case's matrix."""
    f, m, n = c["family"], c["m"], c["n"]
    rows = torch.arange(m, device="cuda")
    if f == "banded":
        lo = (rows - c["hw"]).clamp_(min=0)
        return _window(R, m, n, lo, (rows + c["hw"]).clamp_(max=n - 1) - lo + 1, c["r"])
    if f == "blockdiag":
        lo = rows // c["block"] * c["block"]
        return _window(R, m, n, lo, (n - lo).clamp_(max=c["block"]), c["r"])
    if f == "shortwide":  # runs of at most 48 columns in random 64-wide blocks
        z = torch.randn(m, generator=R.g, device="cuda", dtype=torch.float64)
        L = torch.exp(math.log(c["mean"]) - c["sigma"] ** 2 / 2 + c["sigma"] * z).round().long()
        L.clamp_(min=1, max=n // 2)
        k = (L + 47) // 48
        blocks = n // 64
        runs = torch.repeat_interleave(rows, k)
        runs = torch.unique(runs * blocks + R.below(blocks, runs.numel()))
        row, block = runs // blocks, runs % blocks
        size = (L[row] + k[row] - 1) // k[row]
        off = (R.uni(runs.numel()) * (65 - size)).long()
        first = row * n + block * 64 + off
        at = torch.cumsum(size, 0) - size
        inside = torch.arange(int(size.sum()), device="cuda") - torch.repeat_interleave(at, size)
        return torch.repeat_interleave(first, size) + inside
    if f == "circuit":  # diagonal, band, long-range columns, a few dense rows
        K = _powerlaw(R.uni(m), 3.0, 1.0, 1000.0).ceil().long().clamp_(max=n)
        dense = torch.randperm(m, generator=R.g, device="cuda")[: max(1, m // 10_000)]
        longest = max(1, n * 2 // 11)
        length = _powerlaw(R.uni(dense.numel()), 3.0, min(1000.0, float(longest)), float(longest))
        length[0] = longest
        K[dense] = length.long()
        is_dense = torch.zeros(m, dtype=torch.bool, device="cuda")
        is_dense[dense] = True
        d = torch.arange(-8, 9, device="cuda")
        keep = torch.rand(m, 17, generator=R.g, device="cuda") < 0.43
        keep[:, 8] = True
        keep &= ~is_dense[:, None]
        col = rows[:, None] + d[None, :]
        keep &= (col >= 0) & (col < n)
        row, band = keep.nonzero(as_tuple=True)
        far = torch.repeat_interleave(rows, K)
        return torch.unique(torch.cat([row * n + row + band - 8,
                                       far * n + R.below(n, far.numel())]))
    if f == "powerlaw":
        L = _powerlaw(R.uni(m), c["expo"], c["lmin"], c["lmax"] + 1.0).floor().long()
    elif f == "plfamily":
        top = float(min(n, 50.0 * c["r"]))
        L = _powerlaw(R.uni(m), c["expo"], gen._pl_xmin(c["expo"], c["r"], top), top).round().long()
    else:  # uniform lengths, some rows empty
        L = R.below(c["lmax"] + 1, m)
        L[R.uni(m) < c["p_empty"]] = 0
    if f != "uniform":
        L.clamp_(min=1)
    L.clamp_(max=n)
    far = torch.repeat_interleave(rows, L)
    return torch.unique(far * n + R.below(n, far.numel()))


def _matrix(c, R):
    """rowptr, col (int32), val (FP64) on the GPU."""
    m, n = c["m"], c["n"]
    keys = _keys(c, R)
    row = keys // n
    rowptr = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.bincount(row, minlength=m), 0, out=rowptr[1:])
    col = (keys - row * n).int()
    unit = c["family"] == "shortwide"
    val = torch.ones(col.numel(), dtype=torch.float64, device="cuda") if unit else R.sym(col.numel())
    return rowptr, col, val


def _mean_nnz(c):
    """Expected nnz of the case's matrix."""
    f, m, n = c["family"], c["m"], c["n"]
    if f == "banded":
        w = 2 * c["hw"] + 1
        q = np.linspace(0.5, 1.5, 201) * c["r"]
        return m * float(np.minimum(np.maximum(q, 1), w).mean())
    if f == "blockdiag":
        q = np.linspace(0.5, 1.5, 201) * c["r"]
        return m * float(np.minimum(np.maximum(q, 1), min(c["block"], n)).mean())
    if f == "circuit":
        return 10.4 * m + m * 0.17
    if f == "shortwide":
        return m * c["mean"]
    if f == "uniform":
        return m * (1 - c["p_empty"]) * c["lmax"] / 2
    u = (np.arange(20_000) + 0.5) / 20_000
    if f == "powerlaw":
        L = np.floor(_powerlaw(u, c["expo"], c["lmin"], c["lmax"] + 1.0))
    else:
        top = float(min(n, 50.0 * c["r"]))
        L = np.round(_powerlaw(u, c["expo"], gen._pl_xmin(c["expo"], c["r"], top), top))
    return m * float((n * -np.expm1(np.minimum(np.maximum(L, 1), n) * math.log1p(-1.0 / n))).mean())


def _batch_cases(c):
    """The matrices of a batch: banded, power-law and block-diagonal families
    in turn, rows and nnz per row spread over their logarithms."""
    out = []
    for i in range(c["count"]):
        g = np.random.default_rng(c["base"] + i)
        n = int(round(math.exp(g.uniform(math.log(c["nmin"]), math.log(c["nmax"])))))
        r = float(math.exp(g.uniform(math.log(4.0), math.log(200.0))))
        d = dict(m=n, n=n, r=r)
        if i % 3 == 0:
            d.update(family="banded", hw=int(g.integers(1, 65)))
        elif i % 3 == 1:
            d.update(family="plfamily", expo=float(g.uniform(1.6, 3.0)))
        else:
            d.update(family="blockdiag", block=int(g.integers(16, 257)))
        out.append(d)
    return out


def _training(c, seed):
    """Features and class times: the recorded ones, resampled and varied a
    little, as another collection of timings would."""
    D = np.load(os.path.join(selector.DATA_DIR, "train_c5_seed10000_4000.npz"))
    g = np.random.default_rng(seed)
    at = g.permutation(len(D["features"]))[: c["samples"]]
    X = D["features"][at] * (1.0 + 0.01 * g.standard_normal((len(at), 1)))
    t = D["times_ms"][at] * np.exp(0.02 * g.standard_normal((len(at), selector.N_CLASSES)))
    return X.astype(np.float32), t.astype(np.float32)


# ---- preparing and running -------------------------------------------------


def _inputs(c, seed):
    """rowptr (int64), col, val, x, y of one product, FP64, on the GPU."""
    R = _Rand(seed)
    rowptr, col, val = _matrix(c, R)
    return rowptr, col, val, R.sym(c["n"]), R.sym(c["m"])


def _batch_inputs(c, seed):
    cases = _batch_cases(c)
    y = _Rand(seed).sym(sum(d["m"] for d in cases))
    mats, at = [], 0
    for i, d in enumerate(cases):
        R = _Rand(seed * 1009 + i)
        rowptr, col, val = _matrix(d, R)
        mats.append(dict(m=d["m"], n=d["n"], rowptr=rowptr.int(), col=col, val=val,
                         x=R.sym(d["n"]), y=y[at:at + d["m"]], alpha=1.0, beta=c["beta"]))
        at += d["m"]
    return mats, y


def prepare(case, seed):
    c, op = case, case["op"]
    if op == "train":
        X, t = _training(c, seed)
        return dict(case=c, X=X, t=t)
    if op == "batch":
        mats, y = _batch_inputs(c, seed)
        pick = selector.Selector()
        return dict(case=c, y=y, batch=Batch(mats, [pick.select(d) for d in mats]))
    rowptr, col, val, x, y = _inputs(c, seed)
    if op == "host":
        held = [t.cpu().pin_memory() for t in (rowptr, col, val, x, y)]
        s = dict(zip(("rowptr", "col", "val", "x", "y"), (t.numpy() for t in held)))
        return dict(case=c, held=held, nnz=col.numel(), **s)
    rowptr = rowptr.int()
    if op == "once":
        return dict(case=c, rowptr=rowptr, col=col, val=val, x=x, y=y,
                    alpha=ctypes.c_double(c["alpha"]), beta=ctypes.c_double(c["beta"]))
    f32 = c["form"] != "f64"
    if f32:
        val, x = val.float(), x.float()
    plan = Plan(rowptr, col, val, c["n"], kernel=c["kernel"], f32=f32,
                f32_lanes=c["form"] == "lanes")
    return dict(case=c, plan=plan, x=x, y=y)


def run(s):
    c, op = s["case"], s["case"]["op"]
    if op == "spmv":
        s["plan"].spmv(s["x"], s["y"], c["alpha"], c["beta"])
        return s["y"]
    if op == "batch":
        s["batch"].run_graph()
        return s["y"]
    if op == "train":
        return selector.train(s["X"], s["t"], steps=c["steps"])
    if op == "once":
        if c["entry"] == "csr5":
            rc = sbb.lib().csr5_kernel(c["m"], c["n"], s["col"].numel(), ctypes.byref(s["alpha"]),
                                       s["val"].data_ptr(), s["rowptr"].data_ptr(),
                                       s["col"].data_ptr(), s["x"].data_ptr(),
                                       ctypes.byref(s["beta"]), s["y"].data_ptr())
            if rc != 0:
                raise RuntimeError(sbb.last_error())
            return s["y"]
        plan = Plan(s["rowptr"], s["col"], s["val"], c["n"], kernel=c["entry"])
        plan.spmv(s["x"], s["y"], c["alpha"], c["beta"])
        plan.close()
        return s["y"]
    args = (c["m"], c["n"], s["nnz"], c["alpha"], s["val"], s["rowptr"], s["col"], s["x"],
            c["beta"], s["y"])
    if c["entry"] == "baseline":
        rc = api.spMV_mgpu_baseline(*args)
    elif c["entry"] == "v1":
        rc = api.spMV_mgpu_v1(*args, kernel=c["kernel"])
    else:
        rc = api.spMV_mgpu_v2(*args, kernel=c["kernel"], nb=max(1, s["nnz"] // c["tasks"]),
                              q=c["q"])
    if rc != 0:
        raise RuntimeError(sbb.last_error())
    return s["y"]


# ---- what a pass needs, and its outputs in 64 bits -------------------------


def _product_bytes(c, per_nnz, per_row, per_x):
    y = 8 if c["beta"] == 0.0 else 16
    return per_nnz * _mean_nnz(c) + per_row * (c["m"] + 1) + per_x * c["n"] + y * c["m"]


def work(case):
    c, op = case, case["op"]
    if op == "train":
        per = 12 * 64 + 64 * 64 + 64 * 6  # weights: a multiply-add each, forward and twice backward
        return dict(bytes=4 * c["samples"] * (12 + 6 + 1) + 8 * selector.N_PARAMS + 4 * c["steps"],
                    flops=6 * per * c["samples"] * c["steps"])
    if op == "batch":
        every = [dict(d, beta=c["beta"]) for d in _batch_cases(c)]
        return dict(bytes=sum(_product_bytes(d, 12, 4, 8) for d in every),
                    flops=sum(2 * _mean_nnz(d) + 3 * d["m"] for d in every))
    flops = 2 * _mean_nnz(c) + 3 * c["m"]
    if op == "spmv" and c["form"] != "f64":
        return dict(bytes=_product_bytes(c, 8, 4, 4), flops=flops)
    return dict(bytes=_product_bytes(c, 12, 8 if op == "host" else 4, 8), flops=flops)


def _product(rowptr, col, val, x, y, alpha, beta):
    row = torch.repeat_interleave(torch.arange(y.numel(), device=y.device), rowptr.diff().long())
    ax = torch.zeros_like(y).index_add_(0, row, val.double() * x.double()[col.long()])
    return alpha * ax if beta == 0.0 else alpha * ax + beta * y


def _exact_training(c, seed):
    X, t = _training(c, seed)
    P = torch.from_numpy(selector.init_params(X, 0)).double()
    Xd, T, W = (torch.from_numpy(np.asarray(a)).double()
                for a in (X, selector.targets(t), selector.sample_weights(t)))
    lr, wd = float(np.float32(3e-3)), float(np.float32(1e-4))
    fixed = 2 * selector.N_FEATURES
    m, v, hist = torch.zeros_like(P), torch.zeros_like(P), []
    for k in range(1, c["steps"] + 1):
        p = P.clone().requires_grad_(True)
        w = {}
        for name, shape in (("mu", (12,)), ("sd", (12,)), ("W1", (64, 12)), ("b1", (64,)),
                            ("W2", (64, 64)), ("b2", (64,)), ("W3", (6, 64)), ("b3", (6,))):
            at = selector.OFF[name]
            w[name] = p[at:at + math.prod(shape)].reshape(shape)
        h = (Xd - w["mu"]) / w["sd"]
        h = torch.relu(h @ w["W1"].T + w["b1"])
        h = torch.relu(h @ w["W2"].T + w["b2"])
        loss = (((h @ w["W3"].T + w["b3"] - T) ** 2).sum(1) * W).sum() / (6 * W.sum())
        loss.backward()
        hist.append(float(loss.detach()))
        g = p.grad + wd * P
        g[:fixed] = 0
        m = 0.9 * m + 0.1 * g
        v = 0.999 * v + 0.001 * g * g
        P = P - lr * (m / (1 - 0.9 ** k)) / ((v / (1 - 0.999 ** k)).sqrt() + 1e-8)
    return P.numpy(), np.asarray(hist)


def exact(case, seed):
    c, op = case, case["op"]
    if op == "train":
        return _exact_training(c, seed)
    if op == "batch":
        mats, _ = _batch_inputs(c, seed)
        return torch.cat([_product(d["rowptr"], d["col"], d["val"], d["x"], d["y"], d["alpha"],
                                   d["beta"]) for d in mats])
    rowptr, col, val, x, y = _inputs(c, seed)
    if op == "spmv" and c["form"] != "f64":
        val, x = val.float(), x.float()
    out = _product(rowptr, col, val, x, y, c["alpha"], c["beta"])
    return out.cpu().numpy() if op == "host" else out
