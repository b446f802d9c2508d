"""Whole-token decoding on a B200 against the CPU oracle: identical greedy
tokens."""
import ctypes as C

import numpy as np
import pytest

from vx_b200 import llama

pytestmark = pytest.mark.gpu


def report(got, want, gaps=None):
    got, want = list(got), list(want)
    if got == want:
        return ""
    at = next(i for i, (g, w) in enumerate(zip(got, want)) if g != w)
    gap = "" if gaps is None else ", top-2 logit gap there %.3g" % gaps[at]
    return "first divergence at step %d: got %d, want %d%s" % (
        at, got[at], want[at], gap)


def test_config2_small_llama_100_tokens(oracle):
    """dim 288, 6 layers, 6 heads, hidden 768, vocab 32000, seq 256, seed 42;
    100 greedy tokens from BOS = 1 must equal the CPU program's."""
    flat, offsets = llama.small_f32_weights()
    cfg = oracle.LlamaConfig(288, 768, 6, 6, 6, 32000, 256)
    want, gaps = oracle.llama_generate(cfg, flat, 1, 100, want_gaps=True)
    dec = llama.small_f32_decoder(flat, offsets)
    got = [1]
    tok = dec.step([1])[0]
    got.append(tok)
    for _ in range(99):
        tok = dec.step(None)[0]           # the argmax stays on the GPU
        got.append(tok)
    dec.close()
    assert got == list(want), report(got, want, gaps)


def test_small_llama_logits_close(oracle):
    flat, offsets = llama.small_f32_weights(seed=43)
    cfg = oracle.LlamaConfig(288, 768, 6, 6, 6, 32000, 256)
    kv = 288
    kc = np.zeros((6, 256, kv), np.float32)
    vc = np.zeros_like(kc)
    dec = llama.small_f32_decoder(flat, offsets)
    for pos, tok in enumerate([1, 17, 31999, 5]):
        want = oracle.llama_forward(cfg, flat, kc, vc, tok, pos)
        dec.step([tok])
        got = dec.logits()[0]
        assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
    dec.close()


def nn_host_model(oracle, tensors, cfgd, max_seq):
    return oracle.nn_model_from_tensors(tensors, cfgd, max_seq)


def oracle_generate(oracle, hm, prompt, steps, max_seq, want_gaps=False):
    return oracle.nn_generate(hm, prompt, steps, max_seq, want_gaps=want_gaps)


SMALL_NN = dict(dim=512, hidden=1408, n_layers=4, q_heads=8, kv_heads=4,
                head_dim=64, vocab=4096)


@pytest.mark.parametrize("batch", [1, 4])
def test_nn_decoder_tokens_match_oracle(oracle, batch):
    """A scaled-down std::nn model (bf16, grouped-query heads): a random prompt
    fed token by token, then greedy steps; every sequence of a batch runs its
    own prompt."""
    max_seq = 96
    dec, tensors = llama.nn_bf16_model(max_seq=max_seq, batch=batch, **SMALL_NN)
    hm = nn_host_model(oracle, tensors, SMALL_NN, max_seq)
    rng = np.random.default_rng(8)
    prompts = rng.integers(0, SMALL_NN["vocab"], (batch, 40))
    steps = 24
    got = [[] for _ in range(batch)]
    for p in range(prompts.shape[1]):
        toks = dec.step(list(prompts[:, p]))
    for _ in range(steps):
        for b in range(batch):
            got[b].append(toks[b])
        toks = dec.step(None)
    dec.close()
    for b in range(batch):
        want = oracle_generate(oracle, hm, list(prompts[b]), steps, max_seq)
        assert got[b] == want, "sequence %d: %s" % (b, report(got[b], want))


def test_nn_decoder_keeps_every_device_table_it_reads(oracle):
    """Whatever the model builder put on the GPU stays allocated while the
    decoder lives: small and large blocks that torch hands out afterwards are
    filled with NaN, and the tokens must not change."""
    import torch
    max_seq = 96
    dec, tensors = llama.nn_bf16_model(max_seq=max_seq, batch=1, **SMALL_NN)
    hm = nn_host_model(oracle, tensors, SMALL_NN, max_seq)
    junk = [torch.full((n,), float("nan"), device="cuda")
            for n in (1, 128, 3072, 6144, 1 << 16, 1 << 18, 1 << 20) for _ in range(4)]
    torch.cuda.synchronize()
    prompt = list(np.random.default_rng(9).integers(0, SMALL_NN["vocab"], 20))
    for t in prompt:
        tok = dec.step([int(t)])[0]
    got = []
    for _ in range(16):
        got.append(tok)
        tok = dec.step(None)[0]
    dec.close()
    del junk
    want = oracle_generate(oracle, hm, prompt, 16, max_seq)
    assert got == want, report(got, want)


def test_more_decoders_at_once_than_have_room_in_the_pinned_page(oracle):
    """34 decoders, of which 32 leave their tokens where the host reads them and two are
    copied; rooms given back are used again; none may see another's token."""
    flat, offsets = llama.small_f32_weights()
    cfg = oracle.LlamaConfig(288, 768, 6, 6, 6, 32000, 256)
    want = {t: list(oracle.llama_generate(cfg, flat, t, 4)) for t in (1, 17, 31999)}
    first = [(1, 17, 31999)[i % 3] for i in range(34)]
    decs = [llama.small_f32_decoder(flat, offsets) for _ in first]
    got = [[t] for t in first]
    for step in range(3):
        for d, t, out in zip(decs, first, got):
            out.append(d.step([t] if step == 0 else None)[0])
    for i in (0, 31, 33):
        decs[i].close()
        decs[i] = llama.small_f32_decoder(flat, offsets)
        got[i] = [first[i]]
    for i, d in enumerate(decs):
        while len(got[i]) < 5:
            got[i].append(d.step([first[i]] if len(got[i]) == 1 else None)[0])
    for d in decs:
        d.close()
    for t, out in zip(first, got):
        assert out == want[t][:5], report(out, want[t])


@pytest.mark.parametrize("q_heads,kv_heads", [(4, 4), (4, 2), (8, 2)])
def test_one_launch_step_matches_the_oracle_and_the_separate_kernels(
        oracle, monkeypatch, q_heads, kv_heads):
    """One sequence, bf16 weights and heads of 128 values, VXB_STEP_KERNEL=1:
    every layer of a step runs as one cooperative launch (kept as a measured
    alternative; the chain of kernels is faster). Its tokens must equal the oracle's,
    and its logits the ones of the chain of separate kernels (the projections
    sum in the same order; attention cuts the positions differently)."""
    from vx_b200 import ops
    shape = dict(dim=512, hidden=1408, n_layers=3, q_heads=q_heads,
                 kv_heads=kv_heads, head_dim=128, vocab=4096)
    max_seq = 160
    prompt = list(np.random.default_rng(11).integers(0, shape["vocab"], 70))
    steps = 40

    def run(dec):
        for t in prompt:
            tok = dec.step([int(t)])[0]
        said, logits = [], []
        for _ in range(steps):
            said.append(tok)
            logits.append(dec.logits()[0].copy())
            tok = dec.step(None)[0]
        return said, logits

    monkeypatch.setenv("VXB_STEP_KERNEL", "1")
    dec, tensors = llama.nn_bf16_model(max_seq=max_seq, batch=1, **shape)
    assert dec.kernels_per_step == 0           # nothing recorded yet
    got, got_logits = run(dec)
    assert dec.kernels_per_step <= 5, "the step did not run as one launch"
    assert ops.kernel_status() == 0
    dec.close()
    hm = nn_host_model(oracle, tensors, shape, max_seq)
    want = oracle_generate(oracle, hm, prompt, steps, max_seq)
    assert got == want, report(got, want)

    monkeypatch.setenv("VXB_STEP_KERNEL", "0")
    chain, _ = llama.nn_bf16_model(max_seq=max_seq, batch=1, **shape)
    ref, ref_logits = run(chain)
    assert chain.kernels_per_step > 5
    chain.close()
    assert ref == want
    for a, b in zip(got_logits, ref_logits):
        assert np.abs(a - b).max() <= 1e-5 * np.abs(b).max()


@pytest.mark.parametrize("batch", [1, 2])
def test_kv_cache_handed_from_a_prefill_decoder_to_a_decode_decoder(oracle, batch):
    """The disaggregated prefill/decode of the reference's llama program
    (handoff_kv, tests/backend/pass/llama2.vx:431-458): one decoder reads the
    prompt, its K and V caches travel through vx_plugin_transfer_peer, and a
    second decoder that never saw the prompt goes on from them. The transfer
    carries the result: with zeroed caches handed over the tokens differ."""
    from vx_b200 import abi
    from vx_b200.lib import lib
    max_seq = 96
    pre, tensors = llama.nn_bf16_model(max_seq=max_seq, batch=batch, **SMALL_NN)
    dec, _ = llama.nn_bf16_model(max_seq=max_seq, batch=batch, **SMALL_NN)
    hm = nn_host_model(oracle, tensors, SMALL_NN, max_seq)
    prompts = np.random.default_rng(12).integers(0, SMALL_NN["vocab"], (batch, 30))
    steps = 20
    want = [oracle_generate(oracle, hm, [int(t) for t in prompts[b]], steps, max_seq)
            for b in range(batch)]
    for p in range(prompts.shape[1]):
        first = pre.step([int(t) for t in prompts[:, p]])
    nbytes = pre.kv_cache_bytes
    assert nbytes == dec.kv_cache_bytes == 4 * SMALL_NN["n_layers"] * batch * max_seq * \
        SMALL_NN["kv_heads"] * SMALL_NN["head_dim"]

    def go_on(k, v):
        dec.adopt_kv(k, v, prompts.shape[1])
        got, toks = [[] for _ in range(batch)], list(first)
        for _ in range(steps):
            for b in range(batch):
                got[b].append(toks[b])
            toks = dec.step(toks)
        return got

    here = abi.home_gpu()
    k = lib().vx_plugin_transfer_peer(pre.kv_cache(0), here, here, nbytes)
    v = lib().vx_plugin_transfer_peer(pre.kv_cache(1), here, here, nbytes)
    pre.close()                        # the prefill side is gone: only k, v remain
    got = go_on(k, v)
    lib().vx_plugin_free(k, here)
    lib().vx_plugin_free(v, here)
    for b in range(batch):
        assert got[b] == want[b], "sequence %d: %s" % (b, report(got[b], want[b]))

    zeros = abi.DeviceTensor.from_host(np.zeros(nbytes // 4, np.float32))
    assert go_on(zeros.ptr, zeros.ptr) != want
    zeros.free()
    dec.close()


def test_nn_decoder_with_the_split_attention_kernel(oracle):
    """The decoder recorded while the split kernel is chosen: the partial
    results go through the decoder's scratch and counters instead of a
    cluster's shared memory, and the tokens are still the oracle's."""
    from vx_b200.lib import lib
    max_seq, steps = 96, 16
    before = lib().vx_b200_attention_kernel(2)
    try:
        dec, tensors = llama.nn_bf16_model(max_seq=max_seq, batch=2, **SMALL_NN)
        hm = nn_host_model(oracle, tensors, SMALL_NN, max_seq)
        prompts = np.random.default_rng(9).integers(0, SMALL_NN["vocab"], (2, 40))
        got = [[], []]
        for p in range(prompts.shape[1]):
            toks = dec.step(list(prompts[:, p]))
        for _ in range(steps):
            for b in range(2):
                got[b].append(toks[b])
            toks = dec.step(None)
        dec.close()
    finally:
        lib().vx_b200_attention_kernel(before)
    for b in range(2):
        want = oracle_generate(oracle, hm, list(prompts[b]), steps, max_seq)
        assert got[b] == want, "sequence %d: %s" % (b, report(got[b], want))


WIDE_NN = dict(dim=2048, hidden=2816, n_layers=2, q_heads=16, kv_heads=4,
               head_dim=128, vocab=2048)


@pytest.mark.parametrize("batch,tensor_cores", [(16, True), (8, True), (16, False)])
def test_nn_decoder_many_sequences(oracle, monkeypatch, batch, tensor_cores):
    """8 and 16 sequences of 2048-wide activations. With head_dim 128 the
    projections run on the tensor cores (activations as three bf16 terms);
    VXB_BATCH_MMA=0 keeps them on the FMA kernels, where sixteen such
    sequences exceed the shared memory of the fused RMSNorm and the decoder
    normalises with a kernel of its own. Either way the tokens must be the
    oracle's."""
    monkeypatch.setenv("VXB_BATCH_MMA", "1" if tensor_cores else "0")
    max_seq, steps = 48, 10
    dec, tensors = llama.nn_bf16_model(max_seq=max_seq, batch=batch, **WIDE_NN)
    hm = nn_host_model(oracle, tensors, WIDE_NN, max_seq)
    rng = np.random.default_rng(21)
    prompts = rng.integers(0, WIDE_NN["vocab"], (batch, 12))
    got = [[] for _ in range(batch)]
    for p in range(prompts.shape[1]):
        toks = dec.step(list(prompts[:, p]))
    for _ in range(steps):
        for b in range(batch):
            got[b].append(toks[b])
        toks = dec.step(None)
    dec.close()
    from vx_b200 import ops
    assert ops.kernel_status() == 0
    for b in (0, batch // 2, batch - 1):
        want = oracle_generate(oracle, hm, list(prompts[b]), steps, max_seq)
        assert got[b] == want, "sequence %d: %s" % (b, report(got[b], want))


def test_prefill_a_whole_prompt_at_once(oracle):
    """A 100-token prompt through vx_decoder_prefill (the positions as the rows
    of tensor-core GEMMs, f32 attention over the prompt), then greedy steps:
    the tokens are the oracle's, which feeds the prompt one token at a time.
    Then the same split in two: 40 single steps, and the next 59 positions as
    one pass that starts at position 40."""
    from vx_b200 import ops
    from vx_b200.lib import lib
    max_seq, steps = 128, 12
    dec, tensors = llama.nn_bf16_model(max_seq=max_seq, batch=1, **WIDE_NN)
    hm = nn_host_model(oracle, tensors, WIDE_NN, max_seq)
    prompt = [int(t) for t in
              np.random.default_rng(33).integers(0, WIDE_NN["vocab"], 100)]
    want = oracle_generate(oracle, hm, prompt, steps, max_seq)

    def greedy(tok):
        got = []
        for _ in range(steps):
            got.append(tok)
            tok = dec.step(None)[0]
        return got

    short = (C.c_int32 * 20)(*prompt[:20])
    assert lib().vx_decoder_prefill(dec.handle, short, 20) == 0   # too few: steps
    arr = (C.c_int32 * 99)(*prompt[:-1])
    assert lib().vx_decoder_prefill(dec.handle, arr, 99) == 99
    got = greedy(dec.step([prompt[-1]])[0])
    assert ops.kernel_status() == 0
    assert got == want, report(got, want)

    dec.reset()
    for t in prompt[:40]:
        dec.step([t], fetch=False)
    rest = (C.c_int32 * 59)(*prompt[40:99])
    assert lib().vx_decoder_prefill(dec.handle, rest, 59) == 59
    got = greedy(dec.step([prompt[-1]])[0])
    assert ops.kernel_status() == 0
    assert got == want, report(got, want)

    dec.reset()
    got = greedy(dec.prefill(prompt))
    dec.close()
    assert got == want, report(got, want)


def test_config5_llama7b_shape_100_tokens(oracle):
    """The benchmarked configuration at its own shape: dim 4096, 32 layers, 32
    heads of 128, hidden 11008, vocab 32000, bf16 weights N(0, 0.02^2) from
    seed 7; a 16-token prompt (uniform ids, seed 8) and 100 greedy steps.
    The tokens must equal the CPU restatement's, step for step (identical
    token text across placements is the reference's own check,
    scripts/campaigns/llama/run_perf_matrix.sh:273-292). The oracle runs 116
    steps of 13 GFLOP on the host cores: about a minute."""
    max_seq, steps = 160, 100
    dec, tensors = llama.nn_bf16_model(max_seq=max_seq, batch=1, **llama.LLAMA2_7B)
    prompt = [int(t) for t in
              np.random.default_rng(8).integers(0, llama.LLAMA2_7B["vocab"], 16)]
    tok = None
    for t in prompt:
        tok = dec.step([t])[0]
    got = []
    for _ in range(steps):
        got.append(tok)
        tok = dec.step(None)[0]
    dec.close()
    from vx_b200 import ops
    assert ops.kernel_status() == 0
    hm = nn_host_model(oracle, tensors, llama.LLAMA2_7B, max_seq)
    del tensors
    want, gaps = oracle_generate(oracle, hm, prompt, steps, max_seq,
                                 want_gaps=True)
    assert got == want, report(got, want, gaps)


def test_a_llama2c_checkpoint_file_decodes_like_the_oracle(oracle, tmp_path):
    """The file format the reference's llama programs load (7 int32, then f32
    weights in llama2.c order): written here from seeded weights, read by
    vx_decoder_from_llama2c, and decoded greedily; the tokens are the CPU
    program's."""
    shape = dict(dim=128, hidden=352, n_layers=3, n_heads=4, n_kv_heads=4,
                 vocab=1000, seq_len=64)
    flat, _ = llama.small_f32_weights(seed=77, **shape)
    path = str(tmp_path / "model.bin")
    llama.write_llama2c(path, flat, **shape)
    cfg = oracle.LlamaConfig(128, 352, 3, 4, 4, 1000, 64)
    want = list(oracle.llama_generate(cfg, flat, 1, 40))
    dec = llama.Decoder.from_llama2c(path)
    got, tok = [1], dec.step([1])[0]
    got.append(tok)
    for _ in range(39):
        tok = dec.step(None)[0]
        got.append(tok)
    dec.close()
    assert got == want, report(got, want)


QUANT_NN = dict(dim=512, hidden=1408, n_layers=3, q_heads=8, kv_heads=4,
                head_dim=64, vocab=4096)


@pytest.mark.parametrize("quant", ["fp8", "q4"])
def test_quantised_decoder_tokens_match_oracle(oracle, quant):
    """The decoder with every layer's projections in fp8 or Q4_0 (quantised on
    the GPU from seeded bf16 weights): a random prompt, then greedy steps; the
    oracle decodes the same codes and scales with the restatements of the
    reference's fp8 / q4 kernels."""
    max_seq, steps = 96, 24
    dec, tensors = llama.nn_quant_model(quant, max_seq=max_seq, **QUANT_NN)
    hm = oracle.quant_model_from_tensors(tensors, QUANT_NN, max_seq, quant)
    prompt = [int(t) for t in
              np.random.default_rng(12).integers(0, QUANT_NN["vocab"], 40)]
    tok = None
    for t in prompt:
        tok = dec.step([t])[0]
    got = []
    for _ in range(steps):
        got.append(tok)
        tok = dec.step(None)[0]
    dec.close()
    want = oracle.quant_generate(hm, prompt, steps, max_seq)
    assert got == want, report(got, want)


@pytest.mark.parametrize("quant", ["fp8", "q4"])
def test_quantised_decoder_with_gains_on_an_8_byte_boundary(quant, monkeypatch):
    """The norms' gains as a slice of a larger tensor: the same logits, bit for bit."""
    import torch
    made = llama.Decoder

    def moved(by):
        def decoder(cfg, weights, keep=None):
            g = torch.Generator(device="cuda")
            g.manual_seed(1)
            n, held = cfg.dim, []

            def gains(_):
                t = torch.zeros(n + 8, dtype=torch.bfloat16, device="cuda")
                t[by:by + n] = 1 + 0.1 * torch.randn(n, generator=g, device="cuda")
                held.append(t)
                return t[by:].data_ptr()
            weights = dict(weights, attn_norm=[gains(p) for p in weights["attn_norm"]],
                           ffn_norm=[gains(p) for p in weights["ffn_norm"]],
                           final_norm=gains(weights["final_norm"]))
            torch.cuda.synchronize()
            return made(cfg, weights, keep=(keep, held))
        return decoder
    logits = []
    for by in (0, 4):
        monkeypatch.setattr(llama, "Decoder", moved(by))
        dec, _ = llama.nn_quant_model(quant, max_seq=32, **QUANT_NN)
        for t in (5, 4000, 17):
            dec.step([t])
        logits.append(dec.logits())
        dec.close()
    assert np.isfinite(logits[0]).all() and np.array_equal(*logits)


@pytest.mark.parametrize("quant,route", [("q4", ""), ("q4", "mma"), ("fp8", ""),
                                         ("fp8", "mma")])
def test_prefill_with_quantised_weights(oracle, quant, route, monkeypatch):
    """A 100-token prompt through vx_decoder_prefill of a decoder with Q4_0 or
    fp8 weights, then greedy steps: the oracle's tokens, which come from one
    step per prompt token. Then 37 single steps and the other 62 positions in
    one pass. By both routes: a matrix unpacked to two (Q4_0) or three (fp8) bf16
    terms for the CTA-pair GEMM (the default), and the mma.sync kernels that
    unpack the codes in registers for sixteen positions (VXB_Q4_PREFILL=mma,
    VXB_FP8_PREFILL=mma)."""
    from vx_b200 import ops
    from vx_b200.lib import lib
    if route:
        monkeypatch.setenv("VXB_Q4_PREFILL" if quant == "q4" else "VXB_FP8_PREFILL", route)
    max_seq, steps = 128, 12
    dec, tensors = llama.nn_quant_model(quant, max_seq=max_seq, **WIDE_NN)
    hm = oracle.quant_model_from_tensors(tensors, WIDE_NN, max_seq, quant)
    prompt = [int(t) for t in
              np.random.default_rng(34).integers(0, WIDE_NN["vocab"], 100)]
    want = oracle.quant_generate(hm, prompt, steps, max_seq)

    def greedy(tok):
        got = []
        for _ in range(steps):
            got.append(tok)
            tok = dec.step(None)[0]
        return got

    arr = (C.c_int32 * 99)(*prompt[:-1])
    assert lib().vx_decoder_prefill(dec.handle, arr, 99) == 99
    got = greedy(dec.step([prompt[-1]])[0])
    assert ops.kernel_status() == 0
    assert got == want, report(got, want)

    dec.reset()
    for t in prompt[:37]:
        dec.step([t], fetch=False)
    rest = (C.c_int32 * 62)(*prompt[37:99])
    assert lib().vx_decoder_prefill(dec.handle, rest, 62) == 62
    got = greedy(dec.step([prompt[-1]])[0])
    dec.close()
    assert ops.kernel_status() == 0
    assert got == want, report(got, want)


def test_quantisers_follow_their_definitions(oracle):
    """vx_b200_quantize against numpy: fp8 scale = block amax / 448 and codes
    that decode (by the definition of f8e4m3) to within half a step of w /
    scale; Q4_0 as llama.cpp: d = the value of largest magnitude / -8, code =
    min(15, floor(w / d + 8.5))."""
    import torch
    from vx_b200.lib import lib
    rows, cols = 200, 256
    w = (torch.randn(rows, cols, generator=torch.Generator().manual_seed(5)) * 0.02) \
        .to(torch.bfloat16).cuda()
    wf = w.float().cpu().numpy()
    codes = torch.empty(rows * cols, dtype=torch.uint8, device="cuda")
    scales = torch.empty(2 * 2, dtype=torch.float32, device="cuda")
    assert lib().vx_b200_quantize(2, w.data_ptr(), rows, cols, codes.data_ptr(),
                                  scales.data_ptr()) == 0
    torch.cuda.synchronize()
    s = scales.cpu().numpy().reshape(2, 2)
    c = codes.cpu().numpy().reshape(rows, cols)
    for br in range(2):
        for bc in range(2):
            blk = wf[br * 128:(br + 1) * 128, bc * 128:(bc + 1) * 128]
            assert s[br, bc] == np.float32(np.abs(blk).max() / np.float32(448.0))
    assert not ((c & 127) == 127).any()
    words = np.ascontiguousarray(c).view(np.uint32).reshape(-1)
    # decode every weight by the definition and compare with w: within half an
    # e4m3 step (2^-4 relative) of the scaled value, and exact at the block amax
    ident = np.eye(cols, dtype=np.float32)
    back = np.stack([oracle.quant_dot_f64("fp8", words, s.reshape(-1), ident[j],
                                          rows, cols) for j in range(0, cols, 37)], 1)
    ref = wf[:, 0:cols:37]
    assert np.abs(back - ref).max() <= np.abs(wf).max() / 448 * 16 + 1e-12
    assert np.abs(back - ref).max() <= 0.07 * np.abs(ref).max()

    codes4 = torch.empty(rows * cols // 2, dtype=torch.uint8, device="cuda")
    scales4 = torch.empty(rows * cols // 32, dtype=torch.float16, device="cuda")
    assert lib().vx_b200_quantize(3, w.data_ptr(), rows, cols, codes4.data_ptr(),
                                  scales4.data_ptr()) == 0
    torch.cuda.synchronize()
    g = wf.reshape(-1, 32)
    at = np.abs(g).argmax(1)
    d = g[np.arange(g.shape[0]), at] / np.float32(-8.0)
    assert np.array_equal(scales4.cpu().numpy(), d.astype(np.float16))
    want = np.minimum(15, np.floor(g * (np.float32(1.0) / d)[:, None]
                                   + np.float32(8.5))).astype(np.int64)
    want = np.maximum(want, 0)
    nib = codes4.cpu().numpy().reshape(-1, 16)
    got = np.empty((g.shape[0], 32), np.int64)
    got[:, 0::2] = nib & 15
    got[:, 1::2] = nib >> 4
    assert np.array_equal(got, want)
