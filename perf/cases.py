"""What this library is timed on: products of every size a program hands to it, through its
public calls.

Kinds of case
  dgemm   ``eb.dgemm_device`` on device matrices (padded leading dimensions, transposes,
          alpha / beta), with the a-posteriori accuracy check as the default callers use it, or
          stream-ordered without it;
  sgemm   ``eb.sgemm_device`` on device matrices;
  batch   one ``eb.GroupedPlan.execute`` over thousands of uneven small products (the plan is
          kept by the program, like a CUDA graph);
  trsm    ``dtrsm_`` in place on a device right-hand side (Eigen's triangular solves, LLT and LU);
  host    ``dgemm_`` on pageable host matrices: what Eigen's ``operator*`` calls.

All matrices are column-major.  Entries are u 2^e with u uniform in [-1, 1] and e uniform in
{-r .. r}.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import eigen_b200 as eb

BIG = 4096.0 ** 3  # m n k of the largest drawn product
BATCH_SIDE = 256  # largest side of a product in a batch


def listed():
    return [
        # the smallest products that reach the library: one tile, bound by launch and host latency
        dict(name="dgemm_128", kind="dgemm", ta="N", tb="N", m=128, n=128, k=128, alpha=1.0, beta=0.0, pad=0, r=0, check=True),
        # the size of the plain DGEMM configuration that also runs on the CPU
        dict(name="dgemm_512", kind="dgemm", ta="N", tb="N", m=512, n=512, k=512, alpha=1.0, beta=0.0, pad=0, r=0, check=True),
        # odd sizes with a transposed operand and an update of C, as solvers and regressions call it
        dict(name="dgemm_ragged_tn", kind="dgemm", ta="T", tb="N", m=1000, n=1531, k=777, alpha=1.5, beta=0.5, pad=8, r=0, check=True),
        # the middle of the plain sweep: padded leading dimensions, alpha and beta
        dict(name="dgemm_2048_nt", kind="dgemm", ta="N", tb="T", m=2048, n=2048, k=2048, alpha=1.5, beta=0.5, pad=8, r=0, check=True),
        # stream-ordered call (no check) on entries of widely different size
        dict(name="dgemm_stream", kind="dgemm", ta="N", tb="N", m=4096, n=1024, k=3000, alpha=1.0, beta=0.0, pad=0, r=8, check=False),
        # the headline product
        dict(name="dgemm_8192", kind="dgemm", ta="N", tb="N", m=8192, n=8192, k=8192, alpha=1.0, beta=0.0, pad=0, r=0, check=True),
        # single precision, small and ragged
        dict(name="sgemm_ragged_tn", kind="sgemm", ta="T", tb="N", m=300, n=517, k=1100, alpha=1.5, beta=0.5, pad=8, r=0),
        # single precision, large
        dict(name="sgemm_4096", kind="sgemm", ta="N", tb="N", m=4096, n=4096, k=4096, alpha=1.0, beta=0.0, pad=0, r=0),
        # ten thousand uneven products, sides 3 .. 256, a fifth of them fixed-size cubes
        dict(name="batch_f64", kind="batch", dtype="d", count=10000, side=BATCH_SIDE, cubes=0.2, ta="N", tb="N", mix=1),
        dict(name="batch_f32", kind="batch", dtype="s", count=10000, side=BATCH_SIDE, cubes=0.2, ta="N", tb="N", mix=2),
        # a triangular solve with many right-hand sides
        dict(name="trsm_4096", kind="trsm", side="L", uplo="L", trans="N", diag="N", m=4096, n=2048),
        # Eigen's operator* on ordinary host matrices
        dict(name="host_1024", kind="host", ta="N", tb="N", m=1024, n=1024, k=1024, alpha=1.0, beta=0.0),
    ]


def _size(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]; every other one is made odd."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, v | 1 if rng.random() < 0.5 and v < hi else v)


def _mnk(rng, lo, hi):
    while True:
        m, n, k = (_size(rng, lo, hi) for _ in range(3))
        if float(m) * n * k <= BIG:
            return m, n, k


def draw(rng):
    kind = rng.choice(["dgemm", "dgemm", "dgemm", "sgemm", "sgemm", "batch", "trsm", "host"])
    if kind == "dgemm":
        m, n, k = _mnk(rng, 32, 8192)
        return dict(kind=kind, ta=rng.choice("NT"), tb=rng.choice("NT"), m=m, n=n, k=k, alpha=rng.choice([1.0, 1.5, -1.0]),
                    beta=rng.choice([0.0, 0.5, 1.0]), pad=rng.choice([0, 1, 8]), r=rng.choice([0, 0, 8]),
                    check=rng.random() < 0.7)
    if kind == "sgemm":
        m, n, k = _mnk(rng, 32, 8192)
        return dict(kind=kind, ta=rng.choice("NT"), tb=rng.choice("NT"), m=m, n=n, k=k, alpha=rng.choice([1.0, 1.5, -1.0]),
                    beta=rng.choice([0.0, 0.5, 1.0]), pad=rng.choice([0, 1, 8]), r=0)
    if kind == "batch":
        return dict(kind=kind, dtype=rng.choice("ds"), count=_size(rng, 100, 10000), side=_size(rng, 16, BATCH_SIDE),
                    cubes=rng.choice([0.0, 0.2, 0.6]), ta=rng.choice("NT"), tb=rng.choice("NT"), mix=rng.randrange(1 << 20))
    if kind == "trsm":
        return dict(kind=kind, side=rng.choice("LR"), uplo=rng.choice("LU"), trans=rng.choice("NT"), diag=rng.choice("NU"),
                    m=_size(rng, 64, 4096), n=_size(rng, 64, 4096))
    m, n, k = (_size(rng, 64, 2048) for _ in range(3))
    return dict(kind=kind, ta=rng.choice("NT"), tb=rng.choice("NT"), m=m, n=n, k=k, alpha=1.0, beta=rng.choice([0.0, 1.0]))


# ------------------------------------------------------------------ inputs
def _generator(seed, device):
    return torch.Generator(device=device).manual_seed(1000003 * int(seed) + 17)


def _entries(gen, count, r, dtype, device):
    x = torch.empty(count, dtype=dtype, device=device).uniform_(-1.0, 1.0, generator=gen)
    if r:
        e = torch.randint(-r, r + 1, (count,), generator=gen, device=device)
        x = torch.ldexp(x, e)
    return x


def _matrix(gen, rows, cols, ld, r, dtype, device="cuda"):
    """A rows x cols column-major matrix of leading dimension ld: a (cols, ld) tensor."""
    return _entries(gen, cols * ld, r, dtype, device).view(cols, ld)


def _batch_sizes(case):
    """The (m, n, k) of a batch, from the case alone: log-uniform sides and fixed-size cubes."""
    rng = random.Random(case["mix"])
    top = math.log(case["side"])
    out = []
    for _ in range(case["count"]):
        if rng.random() < case["cubes"]:
            out.append((rng.choice((3, 4, 6, 8)),) * 3)
        else:
            out.append(tuple(int(math.exp(rng.uniform(math.log(3), top))) for _ in range(3)))
    return np.array(out, dtype=np.int64)


def _gemm_inputs(case, seed, dtype, device="cuda"):
    g = _generator(seed, device)
    m, n, k, pad = case["m"], case["n"], case["k"], case.get("pad", 0)
    ar, ac = (m, k) if case["ta"] == "N" else (k, m)
    br, bc = (k, n) if case["tb"] == "N" else (n, k)
    r = case.get("r", 0)
    a = _matrix(g, ar, ac, ar + pad, r, dtype, device)
    b = _matrix(g, br, bc, br + pad, r, dtype, device)
    c = _matrix(g, m, n, m + pad, 0, dtype, device)
    return a, b, c


def _batch_inputs(case, seed):
    g = _generator(seed, "cuda")
    dtype = torch.float64 if case["dtype"] == "d" else torch.float32
    mnk = _batch_sizes(case)
    m, n, k = mnk.T
    # every product's operands one after another, each starting on an element of its own
    ea, eb_, ec = m * k, k * n, m * n
    a, b = (_entries(g, int(e.sum()), 0, dtype, "cuda") for e in (ea, eb_))
    c = torch.zeros(int(ec.sum()), dtype=dtype, device="cuda")
    first = [np.concatenate([[0], np.cumsum(e)[:-1]]) for e in (ea, eb_, ec)]
    return mnk, a, b, c, first


def _triangle(case, seed):
    """A well-conditioned triangular matrix of the solve's order (column-major) and B."""
    g = _generator(seed, "cuda")
    s = case["m"] if case["side"] == "L" else case["n"]
    a = _entries(g, s * s, 0, torch.float64, "cuda").view(s, s) / math.sqrt(s)
    a.diagonal().uniform_(1.0, 2.0, generator=g)
    return a, _matrix(g, case["m"], case["n"], case["m"], 0, torch.float64)


# ------------------------------------------------------------------ what a program holds, one pass
def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind in ("dgemm", "sgemm"):
        a, b, c = _gemm_inputs(case, seed, torch.float64 if kind == "dgemm" else torch.float32)
        s.update(a=a, b=b, c0=c if case["beta"] else None, c=c.clone() if case["beta"] else torch.empty_like(c).zero_())
    elif kind == "batch":
        mnk, a, b, c, first = _batch_inputs(case, seed)
        size = a.element_size()
        arr = (eb.GemmProblem * case["count"])()
        q = np.frombuffer(arr, dtype=np.dtype(eb.GemmProblem))
        m, n, k = mnk.T
        q["transa"], q["transb"] = case["ta"].encode(), case["tb"].encode()
        q["m"], q["n"], q["k"] = m, n, k
        q["alpha"], q["beta"] = 1.0, 0.0
        q["lda"] = m if case["ta"] == "N" else k
        q["ldb"] = k if case["tb"] == "N" else n
        q["ldc"] = m
        for f, x, o in zip("abc", (a, b, c), first):
            q[f] = np.uint64(x.data_ptr()) + (o * size).astype(np.uint64)
        s.update(a=a, b=b, c=c, plan=eb.GroupedPlan(case["dtype"], arr))
    elif kind == "trsm":
        a, b = _triangle(case, seed)
        s.update(a=a, b=b, x=b.clone())
    else:
        a, b, c = _gemm_inputs(case, seed, torch.float64, "cpu")
        s.update(a=a.numpy(), b=b.numpy(), c0=c.numpy() if case["beta"] else None, c=c.numpy().copy())
    return s


def run(s):
    q = s["case"]
    kind = q["kind"]
    if kind == "dgemm" or kind == "sgemm":
        a, b, c = s["a"], s["b"], s["c"]
        if s["c0"] is not None:
            c.copy_(s["c0"])  # the C that the product updates
        args = (q["ta"], q["tb"], q["m"], q["n"], q["k"], q["alpha"], a, a.shape[1], b, b.shape[1], q["beta"], c, c.shape[1])
        if kind == "dgemm":
            rc = eb.dgemm_device(*args, check_accuracy=q["check"])
        else:
            rc = eb.sgemm_device(*args)
        if rc != eb.EB2_OK:
            raise RuntimeError(eb.last_error()[1])
        return c[:, : q["m"]]
    if kind == "batch":
        if s["plan"].execute() != eb.EB2_OK:
            raise RuntimeError(eb.last_error()[1])
        return s["c"]
    if kind == "trsm":
        x = s["x"].copy_(s["b"])
        torch.cuda.current_stream().synchronize()  # the BLAS calls run on a stream of their own
        order = q["m"] if q["side"] == "L" else q["n"]
        eb.level3("dtrsm", q["side"], q["uplo"], q["trans"], q["diag"], q["m"], q["n"], 1.0, s["a"], order, x, q["m"])
        return x
    c = s["c"]
    if s["c0"] is not None:
        np.copyto(c, s["c0"])
    eb.dgemm(q["ta"], q["tb"], q["m"], q["n"], q["k"], q["alpha"], s["a"], s["a"].shape[1], s["b"], s["b"].shape[1],
             q["beta"], c, q["m"])
    return c


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind == "batch":
        m, n, k = _batch_sizes(case).astype(float).T
        size = 8 if case["dtype"] == "d" else 4
        return dict(bytes=float(size * (m * k + k * n + m * n).sum()), flops=float((2 * m * n * k).sum()))
    m, n = float(case["m"]), float(case["n"])
    if kind == "trsm":
        s = m if case["side"] == "L" else n
        # run() fills the right-hand side too: B read and written once more
        return dict(bytes=8 * (s * s / 2 + 4 * m * n), flops=m * n * s)
    k = float(case["k"])
    size = 4 if kind == "sgemm" else 8
    # with beta, C is filled before the product, and read by it
    return dict(bytes=size * (m * k + k * n + m * n * (4 if case["beta"] else 1)), flops=2 * m * n * k)


def tolerance(case):
    # four times what another order of the same sums shows: FP32 sums over K = 8192 by FFMA are
    # 1.6e-6 off, FP64 products up to 3e-15 (against another library's order), solves 4e-16
    if case["kind"] == "sgemm" or case.get("dtype") == "s":
        return {"rel": 6.4e-6}
    if case["kind"] == "trsm":
        return {"rel": 4e-15}
    return {"rel": 1.2e-14}


# ------------------------------------------------------------------ the same in 64 bits
def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        mnk, a, b, c, first = _batch_inputs(case, seed)
        a, b = a.double().cpu().numpy(), b.double().cpu().numpy()
        out = np.zeros(c.numel())
        for (m, n, k), oa, ob, oc in zip(mnk.tolist(), *(f.tolist() for f in first)):
            x, y = a[oa:oa + m * k], b[ob:ob + k * n]
            # row-major views of the column-major operands: C^T = op(B)^T op(A)^T
            x = x.reshape(k, m) if case["ta"] == "N" else x.reshape(m, k).T
            y = y.reshape(n, k) if case["tb"] == "N" else y.reshape(k, n).T
            out[oc:oc + m * n] = (y @ x).reshape(-1)
        return torch.from_numpy(out)
    if kind == "trsm":
        a, b = _triangle(case, seed)
        # column-major storage: the tensors are the transposes
        upper = case["uplo"] == "U"
        mat = a.T if case["trans"] == "N" else a
        up = upper if case["trans"] == "N" else not upper
        x = torch.linalg.solve_triangular(mat, b.T, upper=up, left=case["side"] == "L", unitriangular=case["diag"] == "U")
        return x.T.contiguous()
    dev = "cpu" if kind == "host" else "cuda"
    a, b, c = _gemm_inputs(case, seed, torch.float32 if kind == "sgemm" else torch.float64, dev)
    m, n, k = case["m"], case["n"], case["k"]
    a, b, c = (x.double() for x in (a, b, c))
    at = a[:, :m] if case["ta"] == "N" else a[:, :k].T  # op(A)^T, k x m
    bt = b[:, :k] if case["tb"] == "N" else b[:, :n].T  # op(B)^T, n x k
    out = case["alpha"] * (bt @ at)
    if case["beta"]:
        out += case["beta"] * c[:, :m]
    return out if kind != "host" else out.numpy()
