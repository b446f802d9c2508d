"""Products whose sizes and strides fit no tile, on the tensor cores: f32 with the terms
made inside the kernel, 16-bit with operands copied to aligned rows and with the blocks
of K cut into runs."""
import numpy as np
import pytest

from vx_b200 import abi, ops

pytestmark = pytest.mark.gpu


def product(a, b, m, n, k, elem, bf16=False, offsets=(0, 0, 0), pads=(0, 0, 0)):
    """C of m x n from views of A and B that begin `offset` elements into rows `pad`
    elements longer than they need; checks that C's surroundings stay."""
    held = []
    for x, (r, c), off, pad in ((a, (m, k), offsets[0], pads[0]),
                                (b, (k, n), offsets[1], pads[1]),
                                (None, (m, n), offsets[2], pads[2])):
        big = np.full(off + r * (c + pad), 7, a.dtype)
        if x is not None:
            for i in range(r):
                big[off + i * (c + pad): off + i * (c + pad) + c] = x[i]
        held.append((abi.DeviceTensor.from_host(big, bf16=bf16), c + pad, off, (r, c)))
    descs = [abi.descriptor(t.ptr, shape, strides=(ld, 1), offset=off)
             for t, ld, off, shape in held]
    blob = abi.payload("k", abi=1, kind="matmul", roles="a:0,b:1,out:2",
                       outkind="buffer", topo=abi.gpu(0))
    abi.dispatch(blob, descs, [abi.memref_tag(elem, 2)] * 3)
    assert ops.kernel_status() == 0
    t, ld, off, _ = held[2]
    flat = t.to_host()
    for x, *_ in held:
        x.free()
    rows = flat[off:].reshape(m, ld)
    assert np.all(flat[:off] == 7) and np.all(rows[:, n:] == 7)
    return rows[:, :n]


def rel(got, want):
    return np.linalg.norm(got.astype(np.float64) - want) / np.linalg.norm(want)


# edges of the 128 x 128 x 64 tiles, of the two-block segments (128 of K), of the runs
# that 2, 4 and 8 blocks of a cluster take, and views off the 16- and 8-byte grids
F32 = [(1, 1, 1, 0, 0), (128, 128, 64, 0, 0), (129, 127, 65, 0, 0), (257, 300, 190, 2, 0),
       (130, 70, 513, 1, 3), (64, 64, 64 * 9, 0, 2), (100, 100, 64 * 17, 4, 4),
       (33, 4, 64 * 72 + 1, 3, 1), (1500, 1300, 40, 0, 0), (700, 1, 900, 0, 0)]


@pytest.mark.parametrize("m,n,k,off,pad", F32)
def test_f32_products_of_any_shape(m, n, k, off, pad):
    """The sums of 128 of K, in the tensor core, and their f32 total: within 1e-6 of an
    f64 product (the f32 kernel's own bound in this suite is 2e-6), with values that differ
    by twelve orders of magnitude."""
    rng = np.random.default_rng(m + n + k)
    a = (rng.uniform(-1, 1, (m, k)) * 10.0 ** rng.uniform(-6, 6, (m, 1))).astype(np.float32)
    b = (rng.uniform(-1, 1, (k, n)) * 10.0 ** rng.uniform(-6, 6, (1, n))).astype(np.float32)
    got = product(a, b, m, n, k, abi.F32, offsets=(off, off, off), pads=(pad, pad, pad))
    want = a.astype(np.float64) @ b.astype(np.float64)
    scale = np.sqrt((a.astype(np.float64) ** 2).sum(1))[:, None] * \
        np.sqrt((b.astype(np.float64) ** 2).sum(0))[None, :]
    assert np.abs((got - want) / scale).max() <= 1e-6


# edges of the 32 x 32 tiles, of the 8, 32 and 128 of K between sums, of the runs of 2, 4
# and 8 blocks, rows off the 16- and 8-byte grids, and with more blocks than fit at once
SMALL = [(1, 1, 1, 0, 0), (31, 33, 3, 1, 0), (32, 32, 128, 0, 0), (33, 65, 129, 0, 1),
         (64, 31, 256, 2, 2), (257, 300, 190, 0, 0), (8, 40, 3001, 4, 4), (70, 96, 1023, 0, 0),
         (200, 100, 512, 3, 1), (512, 512, 100, 0, 0)]


@pytest.mark.parametrize("m,n,k,off,pad", SMALL)
def test_f32_products_in_small_tiles(m, n, k, off, pad):
    """A sum of four products (four roundings), two of those (one), the sum of these sums with
    its rest (one, where eight products are more than what is there already) and the last
    one: seven roundings of at most 2^-24 of the sum of magnitudes, and what the rest's own
    sum loses, 2^-24 of 2^-24 of it for each eight of K."""
    rng = np.random.default_rng(m * n + k)
    a = rng.uniform(-1, 1, (m, k)).astype(np.float32)
    b = (rng.uniform(-1, 1, (k, n)) * 10.0 ** rng.uniform(-3, 3, (k, 1))).astype(np.float32)
    got = product(a, b, m, n, k, abi.F32, offsets=(off, off, off), pads=(pad, pad, pad))
    want = a.astype(np.float64) @ b.astype(np.float64)
    size = np.abs(a).astype(np.float64) @ np.abs(b).astype(np.float64)
    assert (np.abs(got - want) <= (7 + k / 8 * 2.0 ** -24) * 2.0 ** -24 * size).all()


@pytest.mark.parametrize("m,n,k,off,pad", SMALL)
@pytest.mark.parametrize("order", ["growing", "cancelling"])
def test_f32_small_tiles_whose_sums_grow_or_cancel(order, m, n, k, off, pad):
    """Each eight products larger than all before them, or the second half of K taking the
    first half's sum away: the same seven roundings."""
    rng = np.random.default_rng(m * n + k)
    a = rng.uniform(0.5, 1, (m, k)).astype(np.float32)
    b = rng.uniform(0.5, 1, (k, n)).astype(np.float32)
    at = np.arange(k)[:, None]
    if order == "growing":
        b = (b * 1.5 ** np.minimum(at % 128 // 4, 60)).astype(np.float32)
    else:
        half = k // 2
        a[:, half:2 * half] = a[:, :half]
        b[half:2 * half] = -b[:half] * np.float32(1 + 1e-5)
    got = product(a, b, m, n, k, abi.F32, offsets=(off, off, off), pads=(pad, pad, pad))
    want = a.astype(np.float64) @ b.astype(np.float64)
    size = np.abs(a).astype(np.float64) @ np.abs(b).astype(np.float64)
    assert (np.abs(got - want) <= (7 + k / 8 * 2.0 ** -24) * 2.0 ** -24 * size).all()


# the 128 x 128 tiles alone and in clusters of two, four and eight
@pytest.mark.parametrize("m,n,k", [(1030, 520, 577), (1500, 1500, 130), (600, 600, 641),
                                   (330, 300, 2500)])
def test_f32_products_in_large_tiles(m, n, k):
    rng = np.random.default_rng(k)
    a = rng.uniform(-1, 1, (m, k)).astype(np.float32)
    b = rng.uniform(-1, 1, (k, n)).astype(np.float32)
    got = product(a, b, m, n, k, abi.F32)
    want = a.astype(np.float64) @ b.astype(np.float64)
    scale = np.sqrt((a.astype(np.float64) ** 2).sum(1))[:, None] * \
        np.sqrt((b.astype(np.float64) ** 2).sum(0))[None, :]
    assert np.abs((got - want) / scale).max() <= 1e-6


@pytest.mark.parametrize("k", [150, 1100])
def test_f32_values_that_three_bf16_terms_cannot_carry(k):
    """Infinities, NaN, values whose terms' products would overflow, and values below the
    bf16 range: as plain f32 multiply-adds give them."""
    rng = np.random.default_rng(k)
    m, n = 200, 140
    a = rng.uniform(-1, 1, (m, k)).astype(np.float32)
    b = rng.uniform(-1, 1, (k, n)).astype(np.float32)
    a[3, 5] = np.inf
    b[9, 17] = np.nan
    a[150, 7], b[7, 3] = 1e30, 1e30          # the product overflows to one infinity
    a[199] = rng.uniform(1, 2, k) * 1e-38    # a row below the smallest third term
    b[:, 100] = np.abs(b[:, 100])
    got = product(a, b, m, n, k, abi.F32)
    with np.errstate(all="ignore"):
        want = a.astype(np.float64) @ b.astype(np.float64)
        want32 = want.astype(np.float32)
    assert np.array_equal(np.isnan(got), np.isnan(want32))
    assert np.array_equal(np.isposinf(got), np.isposinf(want32))
    assert np.array_equal(np.isneginf(got), np.isneginf(want32))
    # all terms of this sum are of one sign: k roundings, each at most 2^-24 of it
    assert abs(got[199, 100] / want[199, 100] - 1) <= k * 2.0 ** -24
    # (row 199's results are near the smallest normal f32)
    fine = np.isfinite(want32) & (np.arange(m) != 199)[:, None] & (np.abs(want) < 1e20)
    assert np.abs(got[fine] - want[fine]).max() <= k * 2.0 ** -23


# What the time model sends to small tiles, on the terms' kernel: VXB_F32_TENSOR=1 keeps f32
# on the tensor cores.
@pytest.fixture
def on_tensor_cores(monkeypatch):
    monkeypatch.setenv("VXB_F32_TENSOR", "1")


@pytest.mark.parametrize("m,n,k,off,pad", F32)
def test_f32_products_of_any_shape_on_tensor_cores(on_tensor_cores, m, n, k, off, pad):
    test_f32_products_of_any_shape(m, n, k, off, pad)


@pytest.mark.parametrize("k", [150, 1100])
def test_f32_values_that_terms_cannot_carry_on_tensor_cores(on_tensor_cores, k):
    test_f32_values_that_three_bf16_terms_cannot_carry(k)


def test_f32_values_of_every_size_on_tensor_cores(on_tensor_cores):
    test_f32_values_of_every_size_that_terms_carry()


# sizes that go there by themselves: a tile's own K, clusters of two and four, rows off the
# 16- and 8-byte grids
@pytest.mark.parametrize("m,n,k,off,pad", [(600, 600, 641, 1, 1), (1030, 520, 577, 2, 2),
                                           (1300, 1100, 100, 3, 3), (330, 300, 2500, 0, 2)])
def test_f32_large_tiles_of_special_values(m, n, k, off, pad):
    """Infinities, NaN, a product that overflows, a row of subnormals and whole numbers, in
    views off the grid."""
    rng = np.random.default_rng(m + k)
    a = rng.integers(-8, 9, (m, k)).astype(np.float32)
    b = rng.integers(-8, 9, (k, n)).astype(np.float32)
    args = dict(offsets=(off, off, off), pads=(pad, pad, pad))
    want = a.astype(np.float64) @ b.astype(np.float64)
    assert np.array_equal(product(a, b, m, n, k, abi.F32, **args), want)
    a[3, 5], a[m - 1, 0] = np.inf, 1e30
    b[9, 17], b[0, n - 1] = np.nan, 1e30
    a[20] = rng.uniform(-1, 1, k) * 1e-39
    got = product(a, b, m, n, k, abi.F32, **args)
    with np.errstate(all="ignore"):
        want = a.astype(np.float64) @ b.astype(np.float64)
        want32 = want.astype(np.float32)
    assert np.array_equal(np.isnan(got), np.isnan(want32))
    assert np.array_equal(np.isposinf(got), np.isposinf(want32))
    assert np.array_equal(np.isneginf(got), np.isneginf(want32))
    fine = np.isfinite(want32) & (np.abs(want) < 1e20)
    size = np.abs(np.where(np.isfinite(a), a, 0)).astype(np.float64) @ \
        np.abs(np.where(np.isfinite(b), b, 0)).astype(np.float64)
    # a result is rounded once more where it is subnormal
    bound = (1e-6 * size + 2.0 ** -149)[fine]
    assert (np.abs(got[fine] - want[fine]) <= bound).all()


# runs of K (few tiles), copies (odd rows, views off the grid) of A, of B and of both, a C
# whose rows begin anywhere, the plain kernel's sizes, tiles of 128 and of 256 columns
B16 = [(100, 100, 4000, 0, 0), (128, 256, 1000, 0, 0), (129, 257, 777, 0, 0),
       (300, 264, 1032, 1, 0), (300, 264, 1032, 0, 3), (257, 513, 2055, 3, 5),
       (33, 7, 5, 0, 0), (64, 64, 65, 1, 1), (1, 512, 4096, 0, 0), (2050, 1028, 136, 0, 2),
       (1001, 3003, 333, 0, 0)]


@pytest.mark.parametrize("dtype", ["bf16", "f16"])
@pytest.mark.parametrize("m,n,k,off,pad", B16)
def test_16_bit_products_of_any_shape(oracle, dtype, m, n, k, off, pad):
    """Small integers: every sum is exact in f32, in whatever order, so the result is the
    exact sum rounded once."""
    rng = np.random.default_rng(m + n + k)
    a = rng.integers(-3, 4, (m, k)).astype(np.float32)
    b = rng.integers(-2, 3, (k, n)).astype(np.float32)
    exact = (a.astype(np.int64) @ b.astype(np.int64)).astype(np.float32)
    bf16 = dtype == "bf16"
    to = oracle.f32_to_bf16 if bf16 else (lambda x: x.astype(np.float16))
    got = product(to(a), to(b), m, n, k, abi.BF16 if bf16 else abi.F16, bf16,
                  offsets=(off, off, off), pads=(pad, pad, pad))
    assert np.array_equal(got, to(exact))


@pytest.mark.parametrize("k", [65, 128, 129, 193, 1025, 1088, 1537, 2100])
def test_f32_products_whose_tiles_have_all_of_k(k):
    """Eighty tiles: a block each, so that its two sets of accumulators alternate over the
    whole of K, with a last segment of one block and of several."""
    rng = np.random.default_rng(k)
    m, n = 1280, 1021
    a = rng.uniform(-1, 1, (m, k)).astype(np.float32)
    b = rng.uniform(-1, 1, (k, n)).astype(np.float32)
    want = a.astype(np.float64) @ b.astype(np.float64)
    assert rel(product(a, b, m, n, k, abi.F32), want) <= 6e-7


@pytest.mark.parametrize("m,n,k", [(1500, 1300, 1000), (1500, 1300, 130), (257, 300, 190)])
def test_f32_products_of_one_sign(m, n, k):
    """The tensor core cuts every sum off, so that values of one sign all lose: 2.2e-8 a K
    step of 16, over the eight steps of a segment, and the f32 additions of the segments'
    sums, which err to both sides (the FP32 pipe is 4.2e-7 off at 1000 of K)."""
    rng = np.random.default_rng(k)
    a = rng.uniform(0, 1, (m, k)).astype(np.float32)
    b = rng.uniform(0, 1, (k, n)).astype(np.float32)
    want = a.astype(np.float64) @ b.astype(np.float64)
    assert rel(product(a, b, m, n, k, abi.F32), want) <= 1.4 * 8 * 2.2e-8


def test_f32_products_from_several_threads_at_once():
    """Clusters of two, four and eight blocks, whose number on the GPU the first call asks for."""
    import concurrent.futures
    rng = np.random.default_rng(8)
    jobs = []
    for m, n, k in [(1030, 520, 577), (600, 600, 641), (330, 300, 2500), (257, 300, 190)]:
        a = rng.uniform(-1, 1, (m, k)).astype(np.float32)
        b = rng.uniform(-1, 1, (k, n)).astype(np.float32)
        jobs.append((a, b, m, n, k, a.astype(np.float64) @ b.astype(np.float64)))

    def one(i):
        a, b, m, n, k, want = jobs[i % len(jobs)]
        return rel(product(a, b, m, n, k, abi.F32), want)
    with concurrent.futures.ThreadPoolExecutor(8) as pool:
        assert max(pool.map(one, range(32))) <= 1e-6


def microseconds(a, b, m, n, k):
    """Of one product of device tensors, the least of five runs of twenty."""
    import torch
    ta, tb = abi.DeviceTensor.from_host(a), abi.DeviceTensor.from_host(b)
    tc = abi.DeviceTensor.from_host(np.zeros((m, n), np.float32))
    begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    runs = []
    for _ in range(6):
        begin.record()
        for _ in range(20):
            ops.matmul_into(tc, ta, tb)
        end.record()
        torch.cuda.synchronize()
        runs.append(begin.elapsed_time(end) * 50)
    for t in (ta, tb, tc):
        t.free()
    return min(runs[1:])


def test_f32_values_near_the_smallest_cost_nothing():
    """A softmax weight far below its row's maximum is a value near 1e-38: no reason for
    another path. And a value too large for the terms costs its blocks the multiply-adds of
    the FP32 pipe, which are ten times as many cycles as the products, half of it here."""
    rng = np.random.default_rng(5)
    m, n, k = 1000, 1000, 1000
    a = rng.uniform(0, 1, (m, k)).astype(np.float32)
    b = rng.uniform(0, 1, (k, n)).astype(np.float32)
    plain = microseconds(a, b, m, n, k)
    a[a < 0.3] = 1e-38
    a[a < 0.4] = 1e-45
    assert microseconds(a, b, m, n, k) <= 1.3 * plain
    a[0, 0] = 1e30
    assert microseconds(a, b, m, n, k) <= 5 * plain


def test_f32_values_of_every_size_that_terms_carry():
    """Rows and columns from the smallest subnormal up: the terms are exact, so the bound is
    that of ordinary values, and half the smallest subnormal where a result is one."""
    rng = np.random.default_rng(6)
    m, n, k = 150, 140, 300
    a = rng.uniform(1, 2, (m, k)).astype(np.float32)
    b = rng.uniform(-2, 2, (k, n)).astype(np.float32)
    a = (a.astype(np.float64) * 2.0 ** np.linspace(-149, 8, m)[:, None]).astype(np.float32)
    b = (b.astype(np.float64) * 2.0 ** np.linspace(-140, 8, n)[None, :]).astype(np.float32)
    got = product(a, b, m, n, k, abi.F32)
    want = a.astype(np.float64) @ b.astype(np.float64)
    size = np.abs(a).astype(np.float64) @ np.abs(b).astype(np.float64)
    assert np.all(np.abs(got - want) <= 1e-6 * size + 8 * 2.0 ** -150)


# shapes that the time model sends to the terms made beforehand: one run straight to C, and
# three runs whose sums another kernel adds, to rows that begin anywhere
BEFOREHAND = [(3072, 3072, 1024, 0, 0), (3072, 3068, 512, 0, 0), (1792, 1792, 4096, 0, 0),
              (1790, 1788, 4096, 1, 3)]


@pytest.mark.parametrize("m,n,k,off,pad", BEFOREHAND)
def test_f32_products_of_terms_made_beforehand(m, n, k, off, pad):
    """The small products are added first, so that what the tensor core cuts off at a K step,
    at most 2^-24 of the sum, counts only in the k / 16 steps of the largest."""
    rng = np.random.default_rng(m + k)
    for lowest in (-1, 0):
        a = rng.uniform(lowest, 1, (m, k)).astype(np.float32)
        b = rng.uniform(lowest, 1, (k, n)).astype(np.float32)
        got = product(a, b, m, n, k, abi.F32, offsets=(off, off, off), pads=(pad, pad, pad))
        want = a.astype(np.float64) @ b.astype(np.float64)
        assert rel(got, want) <= 1e-6 + 2.0 ** -24 * k / 16


@pytest.mark.parametrize("m,n,k,off,pad", BEFOREHAND)
def test_f32_terms_made_beforehand_of_values_they_cannot_carry(m, n, k, off, pad):
    """Infinities, NaN and values whose products would overflow, in a few rows and columns;
    a row near the smallest f32. As plain f32 multiply-adds give them."""
    rng = np.random.default_rng(m + k + 1)
    a = rng.uniform(-1, 1, (m, k)).astype(np.float32)
    b = rng.uniform(-1, 1, (k, n)).astype(np.float32)
    a[3, 5], a[m - 1, k - 1] = np.inf, 1e25
    b[9, 17], b[7, n - 2] = np.nan, -np.inf
    a[20] = rng.uniform(1, 2, k) * 1e-38
    got = product(a, b, m, n, k, abi.F32, offsets=(off, off, off), pads=(pad, pad, pad))
    with np.errstate(all="ignore"):
        want = (a.astype(np.float64) @ b.astype(np.float64)).astype(np.float32)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(np.isposinf(got), np.isposinf(want))
    assert np.array_equal(np.isneginf(got), np.isneginf(want))
    fine = np.isfinite(want)
    size = np.sqrt((np.where(np.isfinite(a), a, 0).astype(np.float64) ** 2).sum(1))[:, None] * \
        np.sqrt((np.where(np.isfinite(b), b, 0).astype(np.float64) ** 2).sum(0))[None, :]
    off_by = np.abs(np.where(fine, got, 0).astype(np.float64) - np.where(fine, want, 0))
    assert (off_by / size).max() <= 1e-6 + 2.0 ** -24 * k / 16


def test_f32_products_of_more_rows_than_tiles_in_a_grid():
    """8.4 million rows: a shape with whole tiles goes where its rows fit."""
    import torch
    m, n, k = 65535 * 128 + 256, 128, 64
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    a = torch.rand((m, k), generator=g, device="cuda")
    b = torch.rand((k, n), generator=g, device="cuda")
    c = torch.zeros((m, n), device="cuda")
    t = [abi.DeviceTensor(x.data_ptr(), tuple(x.shape), abi.F32, abi.home_gpu())
         for x in (c, a, b)]
    torch.cuda.synchronize()
    ops.matmul_into(*t)
    torch.cuda.synchronize()
    for at in (0, 1 << 22, m - 300):
        want = a[at:at + 300].double() @ b.double()
        assert ((c[at:at + 300] - want).norm() / want.norm()).item() <= 1e-6
    assert ops.kernel_status() == 0


def test_f32_products_of_a_long_k():
    """Values of one sign over 26624 of K, terms made beforehand: runs of at most 12288,
    whose sums are cut at each step of 16 by at most 2^-24, where one run would be 7.6e-5
    off."""
    import torch
    m, n, k = 2304, 2048, 26624
    g = torch.Generator(device="cuda")
    g.manual_seed(2)
    a = torch.rand((m, k), generator=g, device="cuda")
    b = torch.rand((k, n), generator=g, device="cuda")
    c = torch.zeros((m, n), device="cuda")
    t = [abi.DeviceTensor(x.data_ptr(), tuple(x.shape), abi.F32, abi.home_gpu())
         for x in (c, a, b)]
    torch.cuda.synchronize()
    ops.matmul_into(*t)
    torch.cuda.synchronize()
    for at in (0, 1000, m - 64):
        want = a[at:at + 64].double() @ b.double()
        assert ((c[at:at + 64] - want).norm() / want.norm()).item() <= 12288 / 16 * 2.0 ** -24
    assert ops.kernel_status() == 0
