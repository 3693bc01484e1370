"""The grouped launch at the edges of its fragments and stages (GPU): sides around 8, 16, 24 and 32,
K around the 4-deep steps and 8-deep stages, every transpose, a leading dimension far past 32 bits
of stage step.  What lies beyond a product in memory is NaN, and C keeps its padding.  FP64 is bit for
bit the native kernel, FP32 within the split-BF16 bound, and both are the bits of every class setting."""
import numpy as np
import pytest
import torch

import eigen_b200 as eb

pytestmark = pytest.mark.gpu

SIDES = [1, 7, 8, 9, 16, 17, 24, 25, 32, 33, 57]
DEPTHS = [1, 3, 4, 5, 8, 9, 15, 16, 17, 40]


@pytest.fixture(autouse=True)
def defaults():
    yield
    eb.set_grouped_classes(-1, -1)
    eb.set_dgemm_method(eb.METHOD_AUTO)


def _problems(dtype, seed, deeper=0):
    rng = np.random.default_rng(seed)
    td = torch.float64 if dtype == "d" else torch.float32
    probs, keep = [], []
    for i, m in enumerate(SIDES):
        for j, n in enumerate(SIDES):
            k = DEPTHS[(3 * i + j) % len(DEPTHS)] + deeper
            ta, tb, pad = "NT"[i % 2], "NT"[j % 2], (i + j) % 3
            ar, ac = (m, k) if ta == "N" else (k, m)
            br, bc = (k, n) if tb == "N" else (n, k)
            nan = float("nan")
            a = torch.full((ac + 1, ar + pad), nan, dtype=td)
            b = torch.full((bc + 1, br + pad), nan, dtype=td)
            a[:ac, :ar] = torch.from_numpy(rng.uniform(-1, 1, (ac, ar)))
            b[:bc, :br] = torch.from_numpy(rng.uniform(-1, 1, (bc, br)))
            c = torch.from_numpy(rng.uniform(-1, 1, (n, m + 2))).to(td)
            alpha, beta = [(1.0, 0.0), (1.5, 0.5), (-0.5, 1.0)][(i + 2 * j) % 3]
            t = dict(a=a.cuda(), b=b.cuda(), c=c.cuda())
            keep.append((t, a, b, c, ar, ac, br, bc))
            probs.append(dict(transa=ta, transb=tb, m=m, n=n, k=k, alpha=alpha, beta=beta, lda=ar + pad, ldb=br + pad,
                              ldc=m + 2, **t))
    return probs, keep


@pytest.mark.parametrize("dtype", ["d", "s"])
def test_edges(dtype):
    results = []
    for classes in ((8, 16), (0, 0), (8, 0), (0, 16)):
        eb.set_grouped_classes(*classes)
        probs, keep = _problems(dtype, 11)
        assert eb.gemm_grouped(dtype, probs) == eb.EB2_OK
        torch.cuda.synchronize()
        results.append([p["c"].clone() for p in probs])
    for other in results[1:]:
        assert all(torch.equal(x, y) for x, y in zip(results[0], other))
    eb.set_dgemm_method(eb.METHOD_NATIVE)
    u = 2.0 ** -53 if dtype == "d" else 2.0 ** -24
    for p, (t, a, b, c, ar, ac, br, bc), got in zip(probs, keep, results[0]):
        m, n, k = p["m"], p["n"], p["k"]
        got = got.cpu()
        assert torch.equal(got[:, m:], c[:, m:]), p
        A, B = a[:ac, :ar].double(), b[:bc, :br].double()
        A = A.T if p["transa"] == "N" else A
        B = B.T if p["transb"] == "N" else B
        exact = p["alpha"] * (A @ B) + p["beta"] * c[:, :m].T.double()
        # FP64: k sums; FP32: the dropped piece products and 8-deep chunks (3 + 8 units), then chunk sums
        terms = (k + 2) if dtype == "d" else (11 + k / 8 + 2)
        bound = terms * u * (abs(p["alpha"]) * (A.abs() @ B.abs()) + abs(p["beta"]) * c[:, :m].T.double().abs())
        assert ((got[:, :m].T.double() - exact).abs() <= 2 * bound).all(), p
        if dtype == "d":
            want = c.cuda()
            assert eb.dgemm_device(p["transa"], p["transb"], m, n, k, p["alpha"], p["a"], p["lda"], p["b"], p["ldb"],
                                   p["beta"], want, p["ldc"]) == eb.EB2_OK
            assert torch.equal(got, want.cpu()), p


@pytest.mark.parametrize("dtype", ["d", "s"])
def test_large_leading_dimension(dtype):
    # a K-contiguous operand whose step of four lines passes 2^31 bytes takes the general copies
    td = torch.float64 if dtype == "d" else torch.float32
    size = 8 if dtype == "d" else 4
    ld = 2 ** 31 // (4 * size) + 3
    k, m, n = 11, 6, 20
    big = torch.zeros((m - 1) * ld + k, dtype=td, device="cuda")
    rows = torch.rand((m, k), dtype=td, device="cuda")
    for i in range(m):
        big[i * ld:i * ld + k] = rows[i]
    b = torch.rand((n, k), dtype=td, device="cuda")
    out = []
    for a, lda in ((big, ld), (rows.contiguous(), k)):
        c = torch.zeros((n, m), dtype=td, device="cuda")
        p = [dict(transa="T", transb="N", m=m, n=n, k=k, a=a, lda=lda, b=b, ldb=k, c=c, ldc=m)]
        assert eb.gemm_grouped(dtype, p) == eb.EB2_OK
        torch.cuda.synchronize()
        out.append(c)
    assert torch.equal(out[0], out[1])


@pytest.mark.parametrize("dtype", ["d", "s"])
@pytest.mark.parametrize("classes", [(8, 16), (0, 0)])
def test_few_and_many_items_agree(dtype, classes):
    # the kernel of a launch of few deep items and that of many: the same bits
    eb.set_grouped_classes(*classes)
    probs, keep = _problems(dtype, 13, 128)
    many = [dict(p, c=p["c"].clone()) for _ in range(30) for p in probs]
    # and that of few items without a 32 x 32 tile
    small = [i for i, p in enumerate(probs) if max(p["m"], p["n"]) <= 16]
    few_small = [dict(probs[i], c=probs[i]["c"].clone()) for i in small]
    assert eb.gemm_grouped(dtype, probs) == eb.EB2_OK
    assert eb.gemm_grouped(dtype, many) == eb.EB2_OK
    assert eb.gemm_grouped(dtype, few_small) == eb.EB2_OK
    torch.cuda.synchronize()
    for i, p in enumerate(many):
        assert torch.equal(p["c"], probs[i % len(probs)]["c"]), i
    for i, p in zip(small, few_small):
        assert torch.equal(p["c"], probs[i]["c"]), i


def _deep(dtype, count, k=8192):
    td = torch.float64 if dtype == "d" else torch.float32
    a = torch.rand((count, k, 32), dtype=td, device="cuda")
    b = torch.rand((count, 32, k), dtype=td, device="cuda")
    c = torch.zeros((count, 32, 32), dtype=td, device="cuda")
    return [dict(m=32, n=32, k=k, a=a[i], lda=32, b=b[i], ldb=k, c=c[i], ldc=32) for i in range(count)]


def _best_ms(run):
    times = []
    for _ in range(8):
        t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t0.record()
        run()
        t1.record()
        torch.cuda.synchronize()
        times.append(t0.elapsed_time(t1))
    return min(times)


def test_few_deep_fp64_items_hide_their_loads():
    # one item per SM: the copies of the stages ahead must cover the latency of memory, so a hundred
    # items whose operands do not fit L2 take about as long as one whose operands do
    one, many = eb.GroupedPlan("d", _deep("d", 1)), eb.GroupedPlan("d", _deep("d", 100))
    t1, t100 = _best_ms(one.execute), _best_ms(many.execute)
    assert t100 < 1.25 * t1, (t1, t100)


def test_one_fp32_product_per_launch_keeps_the_plan_s_pace():
    # a warp per tile in both
    probs = _deep("s", 1)
    arr = eb.problems_array(probs)
    plan = eb.GroupedPlan("s", probs)
    t_plan, t_each = _best_ms(plan.execute), _best_ms(lambda: eb.gemm_each("s", arr))
    assert t_each < 1.2 * t_plan, (t_plan, t_each)  # 1.03; 1.4 with 104 registers
