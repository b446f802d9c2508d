"""The kernels of a decode step at the edges of their plans: the argmax over a cluster of
blocks, and attention with one, two and four blocks per head."""
import numpy as np
import pytest

from vx_b200 import abi, llama, ops

pytestmark = pytest.mark.gpu


def argmax(values):
    logits = abi.DeviceTensor.from_host(values)
    out = abi.DeviceTensor.from_host(np.full(1, -1, np.int32))
    ops.nn_argmax(out, logits, len(values))
    got = int(out.to_host()[0])
    logits.free()
    out.free()
    return got


@pytest.mark.parametrize("n", [1, 33, 4095, 4096, 4099, 32000, 151936])
def test_argmax_of_a_cluster_takes_the_lowest_index_of_the_largest(n):
    rng = np.random.default_rng(n)
    x = rng.standard_normal(n).astype(np.float32)
    for at in sorted({0, n // 8, n // 2, max(0, n - 1)}):
        y = x.copy()
        y[at] = 100.0
        assert argmax(y) == at
        if at + 1 < n:                    # an equal one further on, in another block
            y[n - 1] = 100.0
            assert argmax(y) == at
    assert argmax(np.full(n, -np.inf, np.float32)) == 0
    if n > 2:
        y = x.copy()
        y[n // 2] = np.nan                # larger than nothing
        want = int(np.nanargmax(y))
        assert argmax(y) == want
        y[0] = np.nan                     # nothing is larger than a NaN in first place
        assert argmax(y) == 0


@pytest.mark.parametrize("batch,q_heads,kv_heads", [(8, 16, 16), (16, 16, 16), (4, 32, 8),
                                                    (16, 32, 32)])
def test_blocks_per_head_do_not_change_the_logits(batch, q_heads, kv_heads):
    """16 sequences of equal tokens beside one sequence alone, which takes eight blocks a
    head: the same sums in another order, at positions on both sides of a warp's eight
    rows. Two layers of f32 activations: 64 additions of order 1 in a head's sums, so a few
    units of 2^-24 times 64."""
    shape = dict(dim=q_heads * 128, hidden=256, n_layers=2, q_heads=q_heads,
                 kv_heads=kv_heads, head_dim=128, vocab=512, max_seq=96)
    rng = np.random.default_rng(batch + q_heads)
    tokens = rng.integers(0, 512, 70)
    one, held = llama.nn_bf16_model(batch=1, **shape)
    many, held_too = llama.nn_bf16_model(batch=batch, **shape)
    for i, t in enumerate(tokens):
        one.step([int(t)])
        many.step([int(t)] * batch)
        if i in (0, 7, 8, 33, 69):
            a, b = one.logits(), many.logits()
            scale = np.sqrt((a * a).mean())
            assert np.abs(b - a).max() <= 64 * 64 * 2.0 ** -24 * scale
    one.close()
    many.close()
    del held, held_too


@pytest.mark.parametrize("batch,q_heads,kv_heads", [(4, 32, 32), (8, 32, 32), (16, 32, 32),
                                                    (16, 64, 16)])
def test_blocks_per_head_over_a_long_cache(batch, q_heads, kv_heads):
    """The same keys and values for every sequence, 1500 positions: a block goes round its
    loop of loads many times. Sums of 1500 weights in another order: 2^-24 a term at most,
    and the terms add up to one."""
    import torch
    held, rows = 1500, 1536
    shape = dict(dim=q_heads * 128, hidden=256, n_layers=1, q_heads=q_heads, kv_heads=kv_heads,
                 head_dim=128, vocab=512, max_seq=rows)
    g = torch.Generator(device="cuda")
    g.manual_seed(q_heads)
    cache = [torch.randn((1, 1, rows, kv_heads, 128), generator=g, device="cuda")
             for _ in range(2)]
    got = []
    for b in (1, batch):
        d, weights = llama.nn_bf16_model(batch=b, **shape)
        k, v = (c.expand(1, b, -1, -1, -1).contiguous() for c in cache)
        torch.cuda.synchronize()
        d.adopt_kv(k.data_ptr(), v.data_ptr(), held)
        for step in range(3):
            d.step([step + 1] * b)
        got.append(d.logits())
        d.close()
        del weights
    scale = np.sqrt((got[0] ** 2).mean())
    assert np.abs(got[1] - got[0]).max() <= 1500 * 2.0 ** -24 * scale
    assert ops.kernel_status() == 0
