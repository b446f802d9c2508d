"""A matrix that the call just before has made, read by a projection on the same stream with
nothing between: a product lets the next kernel start while it still stores, so what the
projection fetches ahead of that kernel's end must not be its weights."""
import pytest

from vx_b200 import abi, ops
from vx_b200.lib import lib

pytestmark = pytest.mark.gpu

# m, n, k of the product that makes the matrix (or a table of scales), by the kernel it
# runs on: f32 in small tiles, in large ones, of terms made beforehand; 16 bits on one CTA,
# in runs of K, on pairs
MADE = {"f32": [(96, 512, 200), (1030, 520, 577), (3072, 3072, 1024)],
        "bf16": [(1024, 1024, 1024), (256, 512, 8192), (4096, 4096, 2048)]}
CASES = [("flat",) + s for s in MADE["f32"]] + \
        [(c,) + s for c in ("matvec", "swiglu", "rows", "qkv") for s in MADE["bf16"]] + \
        [("q4", 1024, 128, 2048), ("q4 rows", 1024, 128, 2048), ("fp8", 16, 32, 4000)]


def tensor(t, shape=None):
    import torch
    elem = {torch.float32: abi.F32, torch.bfloat16: abi.BF16, torch.float16: abi.F16,
            torch.int32: abi.I32}[t.dtype]
    return abi.DeviceTensor(t.data_ptr(), tuple(shape or t.shape), elem, abi.home_gpu())


@pytest.mark.parametrize("consumer,m,n,k", CASES)
def test_a_projection_reads_what_the_product_before_it_has_made(consumer, m, n, k):
    """Forty times over, two products' values in turn: as after waiting for the product."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(m + n + k)

    def rand(*shape, dtype=torch.float32):
        return (torch.rand(shape, generator=g, device="cuda") - 0.5).to(dtype)
    dtype = {"flat": torch.float32, "fp8": torch.float32, "q4": torch.float16,
             "q4 rows": torch.float16}.get(consumer, torch.bfloat16)
    a = [rand(m, k, dtype=dtype), rand(m, k, dtype=dtype)]
    b, c = rand(k, n, dtype=dtype), torch.zeros((m, n), dtype=dtype, device="cuda")
    flat = tensor(c, (m * n,))
    rows, cols = m, n
    if consumer in ("q4", "q4 rows"):
        cols = 32 * n
        codes = torch.randint(-2**31, 2**31 - 1, (m * cols // 8,), generator=g, device="cuda",
                              dtype=torch.int32)
    elif consumer == "fp8":
        rows, cols = 128 * m, 128 * n
        codes = torch.randint(0, 2**31 - 1, (rows * cols // 4,), generator=g, device="cuda",
                              dtype=torch.int32) & 0x3f3f3f3f
    count = 19 if consumer in ("rows", "q4 rows") else 1
    x = rand(count, cols)
    times = 40
    y = torch.zeros((times, count, rows), device="cuda")
    bias = rand(rows, dtype=torch.bfloat16)
    vector = tensor(x, (cols,))

    def project(out):
        to = tensor(out, (rows,))
        if consumer == "flat":
            lib().vx_plugin_dispatch_async_flat(out.data_ptr(), x.data_ptr(), c.data_ptr(), cols,
                                                rows)
        elif consumer == "matvec":
            ops.nn_matvec(to, flat, vector, rows, cols)
        elif consumer == "swiglu":
            ops.nn_swiglu(tensor(out, (rows // 2,)), flat, vector, rows // 2, cols)
        elif consumer == "rows":
            ops.nn_matvec_rows(tensor(out), flat, tensor(x), count, rows, cols)
        elif consumer == "qkv":         # heads of 64, half as many of k and of v as of q
            h = rows // 64 // 4
            parts = [tensor(out[0, 64 * at:], (heads, 64))
                     for at, heads in ((0, 2 * h), (2 * h, h), (3 * h, h))]
            ops.nn_qkv(*parts, flat, tensor(bias), vector, 2 * h, h, 64, cols)
        elif consumer == "q4 rows":
            ops.nn_matvec_q4_rows(tensor(out), tensor(codes), flat, tensor(x), count, rows, cols)
        else:
            ops.nn_matvec_quant(consumer, to, tensor(codes), flat, vector, rows, cols)

    want = []
    for i in range(2):
        ops.matmul_into(tensor(c), tensor(a[i]), tensor(b))
        torch.cuda.synchronize()
        project(y[i])
        torch.cuda.synchronize()
        want.append(y[i].clone())
    assert not torch.equal(*want)
    y.zero_()
    torch.cuda.synchronize()
    for i in range(times):
        ops.matmul_into(tensor(c), tensor(a[i % 2]), tensor(b))
        project(y[i])
    torch.cuda.synchronize()
    assert ops.kernel_status() == 0
    for i in range(times):
        assert torch.equal(y[i], want[i % 2]), i


@pytest.mark.parametrize("second", ["one CTA", "pairs", "attention"])
def test_a_kernel_whose_predecessor_takes_longer_than_its_waits(second):
    """The scalar product of two vectors of 4.8 GB is one small tile, a cluster of eight
    blocks that take two seconds. What follows is set up on the other SMs meanwhile, and its
    bounded waits, of about a second, must not have begun."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    long = 1_200_000_000
    a, b = torch.full((1, long), 0.5, device="cuda"), torch.full((long, 1), 2.0, device="cuda")
    c = torch.zeros((1, 1), device="cuda")

    def rand(*shape):
        return (torch.rand(shape, generator=g, device="cuda") - 0.5).bfloat16()
    if second == "attention":
        q, k, v = (rand(1, 2, 512, 128) for _ in range(3))
        out, want = torch.zeros_like(q), torch.zeros_like(q)
    else:
        n = 384 if second == "one CTA" else 4096
        q, k = rand(n, n), rand(n, n)
        out, want = torch.zeros_like(q), torch.zeros_like(q)

    def run(to):
        if second == "attention":
            ops.flash_attention(tensor(q), tensor(k), tensor(v), tensor(to), 128 ** -0.5, True)
        else:
            ops.matmul_into(tensor(to), tensor(q), tensor(k))
    run(want)
    torch.cuda.synchronize()
    began, ended = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    began.record()
    ops.matmul_into(tensor(c), tensor(a), tensor(b))
    run(out)
    ended.record()
    torch.cuda.synchronize()
    assert ops.kernel_status() == 0
    assert began.elapsed_time(ended) > 1200     # else this shows nothing
    assert torch.equal(out, want)
    assert c.item() == long
