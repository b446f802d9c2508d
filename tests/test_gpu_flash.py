"""Flash attention forward on a B200 against the oracle's f32 attention over
bf16-rounded inputs; tolerance 2e-2 max-abs, as the configuration states."""
import numpy as np
import pytest

from vx_b200 import abi, ops

pytestmark = pytest.mark.gpu


def make_qkv(oracle, B, H, S, D):
    out = []
    for seed in (10, 11, 12):
        x = np.random.default_rng(seed).standard_normal((B, H, S, D), dtype=np.float32)
        out.append(oracle.f32_to_bf16(x))
    return out


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("B,H,S", [(1, 2, 128), (1, 3, 256), (2, 2, 384),
                                   (1, 2, 1024), (1, 2, 4096)])
def test_flash_matches_oracle(oracle, B, H, S, causal):
    D = 128
    q, k, v = make_qkv(oracle, B, H, S, D)
    tq, tk, tv = (abi.DeviceTensor.from_host(t, bf16=True) for t in (q, k, v))
    to = abi.DeviceTensor.from_host(np.zeros((B, H, S, D), np.uint16), bf16=True)
    scale = 1.0 / np.sqrt(D)
    ops.flash_attention(tq, tk, tv, to, scale, causal)
    assert ops.kernel_status() == 0
    got = oracle.bf16_to_f32(to.to_host())
    # every 37th row, every 331st at the benchmark's sequence length (a row of
    # the oracle costs S * D products), and the rows at tile edges
    rows = np.unique(np.concatenate([np.arange(0, S, 37 if S <= 1024 else 331),
                                     [0, 63, 64, 127, S - 1]]))
    for b in range(B):
        for h in range(H):
            want = oracle.attention_rows(q[b, h], k[b, h], v[b, h], scale,
                                         causal, rows)
            err = np.abs(got[b, h][rows] - want).max()
            assert err <= 2e-2, (b, h, err)
    for t in (tq, tk, tv, to):
        t.free()


def by_keys_of_64(q, k, v, scale, causal):
    """One head in f64, with the probabilities rounded to bf16 where 64 keys at a time
    round them: against a maximum that begins as that of the first 64 keys and follows
    the row's only when 64 more have outgrown it by 2^8."""
    s = (q @ k.T) * (scale * 1.4426950408889634)
    S = len(s)
    if causal:
        s = np.where(np.arange(S)[None, :] <= np.arange(S)[:, None], s, -np.inf)
    most = s[:, :64].max(1)
    total, out = np.zeros(S), np.zeros((S, q.shape[1]))
    for j in range(0, S, 64):
        big = s[:, j:j + 64].max(1)
        new = np.where(big > most + 8.0, big, most)
        fix = np.exp2(most - new)
        most = new
        p = np.exp2(s[:, j:j + 64] - most[:, None])
        bits = p.astype(np.float32).view(np.uint32).astype(np.uint64)
        bits = (bits + 0x7fff + ((bits >> 16) & 1)) & 0xffff0000
        total = total * fix + p.sum(1)
        out = out * fix[:, None] + bits.astype(np.uint32).view(np.float32) @ v[j:j + 64]
    return out / total[:, None]


def run_flash(oracle, q, k, v, causal):
    tq, tk, tv = (abi.DeviceTensor.from_host(t, bf16=True) for t in (q, k, v))
    to = abi.DeviceTensor.from_host(np.zeros(q.shape, np.uint16), bf16=True)
    ops.flash_attention(tq, tk, tv, to, 1.0 / np.sqrt(q.shape[-1]), causal)
    assert ops.kernel_status() == 0
    got = oracle.bf16_to_f32(to.to_host())
    for t in (tq, tk, tv, to):
        t.free()
    return got


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("H,S", [(2, 128), (2, 384), (2, 1152), (30, 640), (150, 128)])
def test_an_odd_number_of_tiles_rounds_by_64_keys(oracle, H, S, causal):
    """Query tiles by themselves, where each finds an SM, and in pairs with one left over.
    The probabilities' own rounding, 2^-9 of a value, is most of the error, and two
    correct choices of the maximum are 3e-3 apart. With the same choice what is left is a
    rare probability that an f32 score rounds to the other side (one of a hundred, at
    2^-8: 4e-4) and the rounding of the output, 2^-9 / sqrt(3) = 1.2e-3, which is taken
    out by rounding both."""
    q, k, v = make_qkv(oracle, 1, H, S, 128)
    got = run_flash(oracle, q, k, v, causal)
    for h in (0, 1, H - 1):
        f = [oracle.bf16_to_f32(x[0, h]).astype(np.float64) for x in (q, k, v)]
        want = by_keys_of_64(*f, 1.0 / np.sqrt(128), causal).astype(np.float32)
        want = oracle.bf16_to_f32(oracle.f32_to_bf16(want))
        assert np.linalg.norm(got[0, h] - want) / np.linalg.norm(want) <= 8e-4


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("S", [128, 384, 512])
def test_rows_that_outgrow_their_maximum(oracle, S, causal):
    """Keys whose length doubles every 32: the scores of a row grow by far more than 2^8
    in the middle of a tile and from one tile to the next, in CTAs of one and of two query
    tiles. The weights are then those of a few keys, each rounded to bf16 once: 2^-8 of
    the largest value, about 4."""
    q, k, v = make_qkv(oracle, 1, 2, S, 128)
    grown = oracle.bf16_to_f32(k) * (2.0 ** np.minimum(np.arange(S) // 32, 6))[:, None]
    k = oracle.f32_to_bf16(grown.astype(np.float32))
    got = run_flash(oracle, q, k, v, causal)
    rows = np.arange(S)
    for h in range(2):
        want = oracle.attention_rows(q[0, h], k[0, h], v[0, h], 1.0 / np.sqrt(128), causal, rows)
        assert np.abs(got[0, h] - want).max() <= 2e-2
