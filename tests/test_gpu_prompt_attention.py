"""Attention over the positions of a prompt on the tensor cores, at the edges of its
tiles (128 positions, 64 keys), of windows and of rings, against the same sums in f64
and against the steps of one token."""
import numpy as np
import pytest

from oracle import gofilorn as plain
from tests import gofilorn_models as models_of
from vx_b200 import llama, ops

from tests.test_gpu_gofilorn import close, cut, decoder, feed_all, tokens_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,window,rows", [
    (2, 1, 64, 129), (2, 2, 1, 128), (3, 1, 63, 200), (4, 2, 65, 33), (2, 1, 1000, 300),
    (2, 1, 130, 65)])
def test_windows_and_rings(heads, kv_heads, window, rows):
    """Portions of `rows` positions and of single ones; the ring of window + rows wraps
    wherever the window is short."""
    cfg = models_of.config(128, 96, [models_of.layer(heads, kv_heads, 128, window, 0.09, 64),
                                     models_of.layer(heads, kv_heads, 128, 2 * window, 0.2, 64)])
    w = models_of.weights(cfg, seed=window)
    tokens = tokens_for(cfg, 460)
    want = plain.logits(tokens, w, cfg)
    d = decoder(cfg, w, max_seq=460, prefill_rows=rows)
    for sizes in ([rows], [2 * rows + 3, 1, 40]):
        d.reset()
        close(feed_all(d, tokens, cut(460, sizes)), want)
    d.close()
    assert ops.kernel_status() == 0


@pytest.mark.parametrize("q_heads,kv_heads", [(4, 4), (8, 2)])
def test_whole_cache(q_heads, kv_heads):
    """Prompts of lengths on both sides of a tile, and ones that go on from a cache that
    holds positions already, against one step per token. Rounding: sums of at most 400
    values in f32, in two orders, through two layers."""
    shape = dict(dim=q_heads * 128, hidden=256, n_layers=3, q_heads=q_heads,
                 kv_heads=kv_heads, head_dim=128, vocab=512, max_seq=420)
    one, held = llama.nn_bf16_model(**shape)
    many, held_too = llama.nn_bf16_model(**shape)
    tokens = [int(t) for t in np.random.default_rng(q_heads).integers(0, 512, 400)]
    want = []
    for t in tokens:
        one.step([t])
        want.append(one.logits()[0])
    for portions in ([33], [64, 65], [65, 64], [129, 128], [130, 200, 70], [257], [400]):
        many.reset()
        at = 0
        for n in portions:
            many.prefill(tokens[at:at + n])
            at += n
        scale = np.sqrt((want[at - 1] ** 2).mean())
        assert np.abs(many.logits()[0] - want[at - 1]).max() <= 400 * 2.0 ** -23 * scale
    one.close()
    many.close()
    del held, held_too
    assert ops.kernel_status() == 0


@pytest.mark.parametrize("heads,kv_heads,window,rows", [(2, 1, 70, 129), (4, 2, 1000, 460)])
def test_values_that_terms_cannot_carry(heads, kv_heads, window, rows):
    """Keys of about 2^58 in a column that no query looks at and the output matrix scales
    down: the logits are those of ordinary keys, by plain multiply-adds over the ring, with
    the window and the gate."""
    cfg = models_of.config(128, 96, [models_of.layer(heads, kv_heads, 128, window, 0.09, 64)])
    w = models_of.weights(cfg, seed=window)
    column = 37
    w["l0.mix.q"].reshape(heads, 128, -1)[:, column] = 0.0
    w["l0.mix.k"].reshape(kv_heads, 128, -1)[:, column] *= 2.0 ** 58
    w["l0.mix.o"].reshape(-1, heads, 128)[:, :, column] *= 2.0 ** -58
    tokens = tokens_for(cfg, 460)
    want = plain.logits(tokens, w, cfg)
    d = decoder(cfg, w, max_seq=460, prefill_rows=rows)
    for sizes in ([rows], [2 * rows + 3, 1, 40]):
        d.reset()
        close(feed_all(d, tokens, cut(460, sizes)), want)
    d.close()
    assert ops.kernel_status() == 0
