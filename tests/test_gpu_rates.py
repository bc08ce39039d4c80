"""Calls off the sizes that the kernels were tuned at, timed on the device beside a comparable call: a form chosen where another
one is several times faster shows as a ratio, whatever the clock."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def L():
    from ngraph_b200 import lib
    return lib


def stream():
    return torch.cuda.current_stream().cuda_stream


def us(call, run=20):
    """shortest time per call of a run of launches"""
    best = float("inf")
    for _ in range(8):
        first, last = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        first.record()
        for _ in range(run):
            assert call() == 0
        last.record()
        last.synchronize()
        best = min(best, first.elapsed_time(last) * 1000 / run)
    return best


def rows_kernel(L, kind, rows, n):
    x, o = torch.rand(rows * n, device="cuda"), torch.empty(rows * n, device="cuda")
    g, b = torch.rand(n, device="cuda"), torch.rand(n, device="cuda")
    if kind == "softmax":
        return lambda: L.LIB.b200_softmax_rows_f32(x.data_ptr(), o.data_ptr(), rows, n, stream())
    return lambda: L.LIB.b200_layer_norm_rows_f32(x.data_ptr(), g.data_ptr(), b.data_ptr(), o.data_ptr(), rows, n, 1e-5, stream())


@pytest.mark.parametrize("kind,times", [("softmax", 1.8), ("norm", 2.05)])
def test_rows_of_odd_length(L, kind, times):
    """beside rows that move in whole vectors; with generic instead of global accesses 2.4 times as long, otherwise 1.2 and 1.7"""
    assert us(rows_kernel(L, kind, 30000, 1535)) < times * us(rows_kernel(L, kind, 30000, 1532))


def binary(L, n, op=0):
    a, b, o = (torch.rand(n, device="cuda") for _ in range(3))
    return lambda: L.LIB.b200_f32_binary(op, a.data_ptr(), b.data_ptr(), o.data_ptr(), n, stream())


@pytest.mark.parametrize("batch,m,k,n", [(10000, 4, 4, 4), (10000, 33, 1, 1), (2000, 140, 2, 1)])
def test_many_small_products(L, batch, m, k, n):
    """about the elements of an elementwise call; a 32 x 32 x 32 block per product takes seven to fourteen times as long"""
    a, b, o = torch.rand(batch * m * k, device="cuda"), torch.rand(batch * k * n, device="cuda"), torch.empty(batch * m * n, device="cuda")
    t = us(lambda: L.LIB.b200_bmm_f32(a.data_ptr(), b.data_ptr(), o.data_ptr(), batch, m, k, n, stream()))
    assert t < 3.0 * us(binary(L, batch * m * n))


def test_large_elementwise(L):
    """three tensors beside the two that an operand of one element leaves: half as much again, and not twice as long"""
    n = 12 << 20
    a, v, o = torch.rand(n, device="cuda"), torch.rand(1, device="cuda"), torch.empty(n, device="cuda")
    two = us(lambda: L.LIB.b200_f32_binary_periodic(0, a.data_ptr(), v.data_ptr(), o.data_ptr(), n, 1, 0, stream()))
    assert us(binary(L, n)) < 1.9 * two


@pytest.mark.parametrize("n", [10000, 625000])
def test_erf_of_few_elements(L, n):
    """beside the square root of as many: a copy of the table per block made 1.3 and 2 times as much of it"""
    x, o = torch.randn(n, device="cuda").abs(), torch.empty(n, device="cuda")
    t = [us(lambda: L.LIB.b200_f32_unary(op, x.data_ptr(), o.data_ptr(), n, stream())) for op in (10, 8)]
    assert t[0] < 1.25 * t[1]


@pytest.mark.parametrize("m,n,k,wide", [(20, 2432, 3072, 9600), (5760, 30, 4096, 30)])
def test_a_reduction_is_not_split_where_that_is_slower(L, m, n, k, wide):
    """beside a product with the same k-blocks per SM and tiles for all SMs, which is not split: half as much again if this one is"""
    from ngraph_b200 import ops
    a, s = torch.randint(-100, 100, (148 * 128 if wide == n else m, k), device="cuda", dtype=torch.int32).to(torch.int8), torch.ones(1, device="cuda")
    w, o = torch.ones((wide, k), device="cuda", dtype=torch.int8), torch.empty((148 * 128 if wide == n else m) * wide, dtype=torch.uint8, device="cuda")
    t = []
    for rows, cols in ((m, n), (148 * 128, n) if wide == n else (m, wide)):
        x, f, out = a[:rows], w[:cols], o[:rows * cols].view(rows, cols)
        ops.qgemm(x, f, s, torch.uint8, out=out)

        def call():
            ops.qgemm(x, f, s, torch.uint8, out=out)
            return 0
        t.append(us(call))
    assert t[0] < 1.12 * t[1]


@pytest.mark.parametrize("m,n,k,out,at,times", [(4096, 768, 3072, torch.uint8, 0, 1.5), (2048, 2048, 4096, torch.int8, 0, 1.4), (1000, 256, 512, torch.int8, 1, 3.0), (19000, 128, 512, torch.float32, 0, 2.8)])
def test_products_with_a_residual(L, m, n, k, out, at, times):
    """beside the same product without one; residual bytes fetched one by one behind the accumulator: 2.2, 2.1, 4.4 and 3.4 times"""
    from ngraph_b200 import ops
    a = torch.randint(-100, 100, (m, k), device="cuda", dtype=torch.int32).to(torch.int8)
    w, s, o = torch.ones((n, k), device="cuda", dtype=torch.int8), torch.full((1,), 0.01, device="cuda"), torch.empty((m, n), device="cuda", dtype=out)
    r = torch.zeros(m * n + 16, device="cuda", dtype=torch.uint8)[at:at + m * n].view(m, n)
    t = []
    for residual in (r, None):
        def call():
            ops.qgemm(a, w, s, out, sum_in=residual, sum_scale=None if residual is None else s, out=o)
            return 0
        t.append(us(call))
    assert t[0] < times * t[1], t


def test_largest_value_around_the_forms(L):
    """the size up to which one cluster does it costs no more than a little beyond it"""
    import ctypes
    t = {}
    for n in (3 << 18, 1 << 20, (1 << 20) + (1 << 17)):
        x, o = torch.rand(n, device="cuda"), torch.empty(1, device="cuda")
        t[n] = us(lambda: L.LIB.b200_reduce_f32(1, x.data_ptr(), o.data_ptr(), (ctypes.c_int64 * 1)(n), 1, (ctypes.c_int64 * 1)(0), 1, stream()))
    assert t[1 << 20] < 1.15 * t[(1 << 20) + (1 << 17)], t


@pytest.mark.parametrize("rows,inner", [(2, (1 << 30) + 16), (257, 1 << 25)])
def test_the_longest_rows(L, rows, inner):
    """Per-axis Quantize and Dequantize of rows beyond 2^30 elements and of more than 2^33: the rate of one scale per tensor, and its values.
    Element by element, with a division per axis, three times as long."""
    import ctypes
    n = rows * inner
    x, q = torch.empty(n, device="cuda").uniform_(-4, 4), torch.empty(n, dtype=torch.int8, device="cuda")
    s, z = torch.rand(rows, device="cuda") * 0.05 + 0.02, torch.arange(rows, device="cuda").to(torch.int8)

    def quantize(shape, axes, scale, zp):
        return lambda: L.LIB.b200_quantize(x.data_ptr(), scale.data_ptr(), zp.data_ptr(), q.data_ptr(), L.I8, (ctypes.c_int64 * len(shape))(*shape), len(shape),
                                           (ctypes.c_int64 * 1)(*axes), len(axes), 4, stream())

    def dequantize(shape, axes, scale, zp):
        return lambda: L.LIB.b200_dequantize(q.data_ptr(), scale.data_ptr(), zp.data_ptr(), x.data_ptr(), L.I8, (ctypes.c_int64 * len(shape))(*shape), len(shape),
                                             (ctypes.c_int64 * 1)(*axes), len(axes), stream())

    ends = [0, inner - 3, (rows // 2) * inner - 3, (rows - 1) * inner - 3, n - 7]  # the elements around row boundaries and at the ends
    rows_of = torch.cat([torch.arange(e, e + 7, device="cuda") for e in ends])
    idx = rows_of // inner
    assert quantize((rows, inner), (0,), s, z)() == 0
    want = (x[rows_of] / s[idx]).round() + z[idx].float()
    assert torch.equal(q[rows_of], want.clamp(-128, 127).to(torch.int8))
    assert us(quantize((rows, inner), (0,), s, z), 3) < 1.5 * us(quantize((n,), (), s[:1], z[:1]), 3)
    assert dequantize((rows, inner), (0,), s, z)() == 0
    assert torch.equal(x[rows_of], (q[rows_of].int() - z[idx].int()).float() * s[idx])
    assert us(dequantize((rows, inner), (0,), s, z), 3) < 1.5 * us(dequantize((n,), (), s[:1], z[:1]), 3)
