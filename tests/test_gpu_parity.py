"""Parity of the CUDA path with the CPU oracle, through the C ABI, on identical seeded models.

Tolerances: greedy / top-k token ids and candidate index sets must be identical; logits
within max-abs 2e-2 (the bound stated for bf16/fp16; fp32 activations make the measured
difference orders of magnitude smaller, and tighter bounds are asserted where they hold);
top-k values 1e-4, block max 1e-4, block sum 1e-3, materialised block 1e-4
(tests/auto_kv_decode.rs:136-215).
"""
import ctypes

import numpy as np
import pytest

from helpers import gpu_cfg, gpu_model_from_oracle, oracle_cfg, top2_gap

pytestmark = pytest.mark.gpu

LOGIT_TOL = 2e-2


def tol(dtype):
    """Measured bound asserted on logits: fp32 storage differs from the oracle only by summation
    order; with a 16-bit KV cache a last-bit difference before rounding moves a cached value by
    one 16-bit ulp, which shows up around 1e-4.  Both are far inside LOGIT_TOL."""
    return 1e-4 if dtype == "f32" else 1e-3


def _pair(R, O, dims, dtype, seed=5, via="new", **kw):
    """The same model on both sides.  via='new' goes through Model::new (host tensors,
    relayout kernel); via='synth' lets the GPU generate the weights itself."""
    opts = {k: kw.pop(k) for k in ("use_graph", "page_tokens") if k in kw}
    oc = oracle_cfg(O, *dims, dtype=dtype, **kw)
    om = O.Model.synth(oc, seed)
    if via == "new":
        gm = gpu_model_from_oracle(R, O, om, dtype, **opts)
    else:
        gm = R.Model.synthetic(gpu_cfg(R, oc), seed, untied_head=bool(oc.untied), dtype=dtype,
                               activation=oc.activation, **opts)
    return om, gm


SMALL = (256, 640, 2, 128, 64, 2, 320)  # auto_kv_decode.rs:6-28 (vocab 320 = 2 blocks)


@pytest.mark.parametrize("dtype", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("via", ["new", "synth"])
def test_hidden_state_and_logits_match_oracle(R, oracle, dtype, via):
    om, gm = _pair(R, oracle, SMALL, dtype, via=via)
    cache = oracle.Cache(om, kv_round=1)
    toks = [1, 2, 3, 300, 17, 5]
    for i, t in enumerate(toks):
        if i % 2 == 0:
            a, b = gm.decode_token_from_id(t), cache.decode_token_from_id(t)
            np.testing.assert_allclose(a, b, atol=2e-5 if dtype == "f32" else 2e-4, rtol=1e-4)
        else:
            a, b = gm.decode_token_logits_from_id(t), cache.decode_logits(t)
            assert np.abs(a - b).max() < tol(dtype) < LOGIT_TOL
        assert gm.len() == cache.len() == i + 1


@pytest.mark.parametrize("dims,kw", [
    ((128, 384, 2, 64, 48, 3, 777), dict(untied=1)),                 # hd 64, untied head, ragged last block
    ((256, 512, 4, 64, 80, 2, 512), dict(kv_heads=2)),               # GQA 2:1
    ((256, 640, 2, 128, 64, 2, 320), dict(activation=1)),            # LeakyReLU^2 FFN
    ((384, 1000, 3, 128, 200, 2, 1000), dict(page_tokens=16)),       # K = 1000: partial chunk rows, small pages
])
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_shape_variants(R, oracle, dims, kw, dtype):
    om, gm = _pair(R, oracle, dims, dtype, **dict(kw))
    cache = oracle.Cache(om, kv_round=1)
    tok = 3
    for _ in range(12):
        a, b = gm.decode_token_logits_from_id(tok), cache.decode_logits(tok)
        assert np.abs(a - b).max() < tol(dtype)
        tok = int(np.argmax(b))


def test_decode_token_from_hidden_vector(R, oracle):  # Model::decode_token / decode_token_argmax
    om, gm = _pair(R, oracle, SMALL, "f32")
    cache = oracle.Cache(om)
    x = (np.random.default_rng(0).standard_normal(256) * 0.02).astype(np.float32)
    np.testing.assert_allclose(gm.decode_token(x), cache.decode_token(x), atol=2e-5, rtol=1e-4)
    # decode_token_argmax = the same layers, then final norm + tied head + arg-max (lib.rs:306-338)
    y = cache.decode_token(x)
    g = om.tensor(oracle.T_GAMMA_FINAL)
    xn = y * np.float32(1.0 / np.sqrt(np.mean(y * y, dtype=np.float32) + np.float32(1e-5))) * g
    logits = om.tensor(oracle.T_EMBED).reshape(320, 256) @ xn
    assert gm.decode_token_argmax(x) == int(np.argmax(logits))
    assert gm.len() == cache.len() == 2


def test_reference_kv_contracts_on_gpu(R, oracle):  # auto_kv_decode.rs:67-215 with ModelWeights::random
    O = oracle
    oc = oracle_cfg(O, *SMALL)
    om = O.Model.reference_random(oc)
    gm = gpu_model_from_oracle(R, O, om, "f32")
    ctx = R.DecodeContext(gm)
    generated = [1, 2, 3, 4]
    logits, kcf, vcf = om.forward_logits(generated, want_kv=True)
    nxt = int(np.argmax(logits[0]))
    naive = om.forward_logits(generated + [nxt])[0]

    ctx.seed_from_forward_caches(kcf, vcf, 4)
    assert ctx.decode_next_greedy_token(nxt) == int(np.argmax(naive))

    ctx.seed_from_forward_caches(kcf, vcf, 4)
    idxs, vals = ctx.decode_next_topk_candidates(nxt, 4)
    order = sorted(range(oc.vocab), key=lambda i: (-naive[i], i))[:4]
    assert idxs.tolist() == order
    np.testing.assert_allclose(vals, naive[order], atol=1e-4)

    ctx.seed_from_forward_caches(kcf, vcf, 4)
    mx, sm = ctx.decode_next_fullvocab_block_stats(nxt, 0.8)
    for b in range(len(mx)):
        z = naive[b * 256:(b + 1) * 256] / np.float32(0.8)
        assert abs(mx[b] - z.max()) < 1e-4 and abs(sm[b] - np.exp(z - z.max()).sum()) < 1e-3
    np.testing.assert_allclose(ctx.materialize_current_logits_block(1), naive[256:320], atol=1e-4)


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_head_entry_points_match_oracle(R, oracle, dtype):
    om, gm = _pair(R, oracle, (256, 640, 2, 128, 64, 2, 1500), dtype)
    cache = oracle.Cache(om, kv_round=1)
    for t in (1, 2, 3):
        gm.decode_token_from_id(t)
        cache.decode_token_from_id(t)
    assert gm.decode_token_argmax_from_id(7) == cache.decode_token_argmax_from_id(7)
    for k in (1, 4, 32):
        gv, gi = gm.decode_token_topk_from_id(9, k)
        ov, oi = cache.decode_token_topk_from_id(9, k)
        np.testing.assert_array_equal(gi, oi)
        np.testing.assert_allclose(gv, ov, atol=tol(dtype))
    for softcap in (0.0, 0.5):
        gmx, gsm = gm.decode_token_block_stats_from_id(11, 1.25, softcap)
        omx, osm = cache.decode_token_block_stats_from_id(11, 1.25, softcap)
        np.testing.assert_allclose(gmx, omx, atol=tol(dtype))
        np.testing.assert_allclose(gsm, osm, atol=10 * tol(dtype))
        for blk in (0, 5):
            np.testing.assert_allclose(gm.materialize_current_logits_block(blk, softcap),
                                       cache.materialize_current_logits_block(blk, softcap), atol=tol(dtype))
    assert len(gm.materialize_current_logits_block(5)) == 1500 - 5 * 256
    assert np.abs(gm.decode_token_logits_from_id(4, 0.3) - cache.decode_logits(4, 0.3)).max() < tol(dtype)


def test_errors_mirror_reference_asserts(R, oracle):
    om, gm = _pair(R, oracle, (256, 640, 2, 128, 8, 2, 320), "f32")
    with pytest.raises(R.CudaDecodeError, match="token id must fit vocab"):
        gm.decode_token_argmax_from_id(320)
    with pytest.raises(R.CudaDecodeError, match="top_k exceeds"):
        gm.decode_token_topk_from_id(1, 33)
    with pytest.raises(R.CudaDecodeError, match="top_k must be positive"):
        gm.decode_token_topk_from_id(1, 0)
    with pytest.raises(R.CudaDecodeError, match="block_idx out of range"):
        gm.materialize_current_logits_block(2)
    for t in range(8):
        gm.decode_token_from_id(t)
    with pytest.raises(R.CudaDecodeError, match="within cfg.seq"):
        gm.decode_token_from_id(1)
    gm.set_len(100)  # clamped to seq, lib.rs:213-215
    assert gm.len() == 8
    assert R.Model.new(gm.cfg, [], {"gamma_final": np.ones(256), "embed": np.zeros(320 * 256)}) is None


C1 = (512, 1536, 8, 64, 512, 8, 8192)  # tiny rustane LM: fp32, untied head, 8 heads x 64


def test_config1_greedy_tokens_and_logits(R, oracle):
    """32 greedy steps from prompt [1,2,3,4] on the tiny LM: ids identical to the committed
    golden vectors (naive_full_context oracle) and per-step logits within tolerance."""
    import os
    gold = np.load(os.path.join(os.path.dirname(__file__), "golden", "config1_greedy.npz"))
    om, gm = _pair(R, oracle, C1, "f32", seed=0, via="synth", untied=1)
    prompt = [1, 2, 3, 4]
    logits = gm.prefill(prompt)
    assert np.abs(logits - gold["logits"][0]).max() < 1e-4 < LOGIT_TOL
    toks = [int(np.argmax(logits))]
    for step in range(1, 32):
        lg = gm.decode_token_logits_from_id(toks[-1])
        assert np.abs(lg - gold["logits"][step]).max() < 1e-4
        toks.append(int(np.argmax(lg)))
    assert toks == gold["tokens"].tolist()
    # the same through the device-resident loop and through the session
    gm.set_len(4)
    assert gm.decode_steps_greedy(toks[0], 31).tolist() == toks[1:]
    sess = R.InferenceSession(gm, prompt)
    for backend in ("cuda", "naive"):
        out = sess.generate(R.GenerationRequest(decode_backend=backend, steps=32))
        assert out.results[0].sampled == toks
        assert out.decode_selection.mode == ("kv_cache_cuda" if backend == "cuda" else "naive_full_context")


def test_long_context_split_k_fp16(R, oracle):
    """Config-2 geometry (dim 1536, 12 x 128, hidden 4096, vocab 32000, seq 2048, fp16) cut to
    3 layers: 512-token prompt, then sampled and greedy continuation vs the oracle."""
    O = oracle
    dims = (1536, 4096, 12, 128, 2048, 3, 32000)
    om, gm = _pair(R, O, dims, "f16", seed=1, via="synth")
    prompt = O.synth_prompt(1, 32000, 512)
    cache = O.Cache(om, kv_round=1)
    for t in prompt[:-1]:
        cache.decode_token_from_id(int(t))
    ref = cache.decode_logits(int(prompt[-1]))
    got = gm.prefill(prompt)
    assert np.abs(got - ref).max() < 1e-3 < LOGIT_TOL
    tok = int(np.argmax(ref))
    assert top2_gap(ref) > 1e-4
    gpu_ids = gm.decode_steps_greedy(tok, 24).tolist()
    ref_ids, cur = [], tok
    for _ in range(24):
        cur = cache.decode_token_argmax_from_id(cur)
        ref_ids.append(cur)
    assert gpu_ids == ref_ids


@pytest.mark.parametrize("mode", ["topk8", "fullvocab", "topk40"])
def test_sampled_requests_match_oracle(R, oracle, mode):
    O = oracle
    dims = (256, 640, 2, 128, 96, 2, 1500)
    om, gm = _pair(R, O, dims, "bf16", seed=21)
    t, k = {"topk8": (0.8, 8), "fullvocab": (1.0, 0), "topk40": (0.9, 40)}[mode]
    prompt = [5, 6, 7, 8, 9]
    ref, ref_mode = om.generate(prompt, 20, backend=O.BACKEND_KV, temperature=t, top_k=k, samples=3, seed=11, kv_round=1)
    sess = R.InferenceSession(gm, prompt)
    out = sess.generate(R.GenerationRequest("cuda", 20, t, k, 3, 11))
    assert ref_mode == O.MODE_KV and out.decode_selection.mode == "kv_cache_cuda"
    for s in range(3):
        assert out.results[s].sampled == ref[s].tolist()
        assert out.results[s].generated == prompt + ref[s].tolist()
        assert out.results[s].seed == 11 + s


def test_session_determinism_suffix_and_streaming(R, oracle):  # inference.rs:976-1033
    om, gm = _pair(R, oracle, (256, 640, 2, 128, 64, 2, 8192), "f32", seed=9)
    req = R.GenerationRequest("cuda", 8, 0.8, 4, 2, 7)
    sess = R.InferenceSession(gm, [1, 2, 3, 4])
    first, second = sess.generate(req), sess.generate(req)
    assert [r.generated for r in first.results] == [r.generated for r in second.results]

    req = R.GenerationRequest("cuda", 6, 0.8, 4, 2, 17)
    ext = R.InferenceSession(gm, [1, 2, 3]).generate_with_suffix(req, [4, 5])
    fresh = R.InferenceSession(gm, [1, 2, 3, 4, 5]).generate(req)
    assert [r.sampled for r in ext.results] == [r.sampled for r in fresh.results]
    ref, _ = om.generate([1, 2, 3], 6, backend=oracle.BACKEND_KV, temperature=0.8, top_k=4, samples=2, seed=17, suffix=[4, 5])
    assert [r.sampled for r in ext.results] == ref.tolist()

    seen = []
    sess = R.InferenceSession(gm, [1, 2, 3, 4])
    one = R.GenerationRequest("cuda", 6, 0.8, 4, 1, 3)
    streamed = sess.generate_stream_with_suffix(one, [], lambda tok, sampled, generated: seen.append((tok, len(sampled), len(generated))))
    assert [s[0] for s in seen] == streamed.results[0].sampled == sess.generate(one).results[0].sampled
    assert [s[1] for s in seen] == list(range(1, 7)) and seen[-1][2] == 10
    with pytest.raises(ValueError, match="streaming only supports samples=1"):
        sess.generate_stream_with_suffix(req, [], lambda *a: None)
    with pytest.raises(ValueError, match="prompt token id 9000 at position 1 exceeds model vocab 8192"):
        R.InferenceSession(gm, [1, 9000])
    with pytest.raises(ValueError, match="at least one token"):
        R.InferenceSession(gm, [])
    # forced cuda falls back when the window does not fit (inference.rs:487-495)
    long = R.InferenceSession(gm, list(range(1, 61)))
    fb = long.generate(R.GenerationRequest("cuda", 8))
    assert fb.decode_selection.mode == "naive_full_context"
    assert fb.decode_selection.fallback_reason == "requested_length_exceeds_cfg_seq"
    ref, _ = om.generate(list(range(1, 61)), 8, backend=oracle.BACKEND_KV)
    assert fb.results[0].sampled == ref[0].tolist()  # sliding window past cfg.seq


def test_checkpoint_graph_and_synthetic_paths_agree_bitwise(R, oracle, tmp_path):
    cfg = R.Config(256, 640, 2, 128, 64, 2, 1500)
    path = str(tmp_path / "m.rstk")
    R.write_synthetic_checkpoint(path, cfg, dtype="bf16", untied_head=True, seed=13)
    a = R.Model.from_checkpoint(path)
    b = R.Model.synthetic(cfg, 13, untied_head=True, dtype="bf16")
    c = R.Model.synthetic(cfg, 13, untied_head=True, dtype="bf16", use_graph=True)
    la, lb, lc = (m.prefill([3, 1, 4, 1, 5]) for m in (a, b, c))
    np.testing.assert_array_equal(la, lb)
    np.testing.assert_array_equal(lb, lc)
    ia, ib, ic = (m.decode_steps_greedy(9, 20) for m in (a, b, c))
    np.testing.assert_array_equal(ia, ib)
    np.testing.assert_array_equal(ib, ic)
    before = c.kernel_launches()
    c.decode_steps_greedy(int(ic[-1]), 4)
    per_token = (c.kernel_launches() - before - 1) / 4
    # one persistent kernel + arg-max, or embed + 5 per layer + head GEMV + arg-max
    assert per_token in (2, 5 * cfg.nlayers + 3)


MEGA_CASES = [
    # dims, dtype, config extras, model options, prompt length
    ((256, 640, 2, 128, 64, 2, 1500), "bf16", {}, {}, 40),                                  # one tile, one CTA per head
    ((512, 1536, 8, 64, 512, 3, 8192), "f32", dict(kv_heads=4), dict(page_tokens=16), 300),   # fp32 cache, hd 64, two q heads per kv head, 16-token tiles
    ((1536, 4096, 12, 128, 2048, 2, 32000), "f16", {}, dict(page_tokens=16), 1700),           # nine tiles per CTA: several rounds through the ring
    ((1024, 2816, 8, 128, 1024, 2, 32000), "bf16", {}, dict(kv_dtype="bf16"), 700),           # 64-token tiles, bf16 cache
]


@pytest.mark.parametrize("dims,dtype,kw,opts,nprompt", MEGA_CASES)
def test_persistent_kernel_path_matches_oracle(R, oracle, dims, dtype, kw, opts, nprompt):
    """The one-cooperative-kernel-per-token path (the default where its tiling covers the shape) against the
    oracle and against the kernel-per-operator path: the prompt goes through the same prompt pass on both models, then single steps (logits) and a
    greedy run.  The cases cover one and several attention tiles per CTA, 16- and 64-token tiles,
    both head dimensions, grouped q heads and the three cache types."""
    O = oracle
    oc = oracle_cfg(O, *dims, dtype=dtype, **kw)
    om = O.Model.synth(oc, 31)
    if opts.get("kv_dtype") == "bf16":
        om.set_kv_dtype(O.BF16)
    mega = R.Model.synthetic(gpu_cfg(R, oc), 31, dtype=dtype, mega=True, use_graph=True, **opts)
    base = R.Model.synthetic(gpu_cfg(R, oc), 31, dtype=dtype, mega=False, **opts)
    cache = O.Cache(om, kv_round=1)
    prompt = O.synth_prompt(4, oc.vocab, nprompt)
    for t in prompt[:-1]:
        cache.decode_token_from_id(int(t))
    ref = cache.decode_logits(int(prompt[-1]))
    got = mega.prefill(prompt)
    assert np.abs(got - ref).max() < tol(dtype)
    assert np.abs(got - base.prefill(prompt)).max() < tol(dtype)
    tok = int(np.argmax(ref))
    for _ in range(6):  # single steps: logits of the three
        a, b, c = mega.decode_token_logits_from_id(tok), base.decode_token_logits_from_id(tok), cache.decode_logits(tok)
        assert np.abs(a - c).max() < tol(dtype) and np.abs(a - b).max() < tol(dtype)
        tok = int(np.argmax(c))
    before = mega.kernel_launches()
    ids = mega.decode_steps_greedy(tok, 16).tolist()
    assert (mega.kernel_launches() - before - 1) / 16 == 2   # the persistent kernel and the head reduction
    assert ids == base.decode_steps_greedy(tok, 16).tolist()
    cur, want = tok, []
    for _ in range(16):
        lg = cache.decode_logits(cur)
        if top2_gap(lg) < 10 * tol(dtype):
            break
        cur = int(np.argmax(lg))
        want.append(cur)
    assert ids[:len(want)] == want and len(want) >= 4


def test_small_kv_golden_vectors(R):
    """Fixed expectations (tests/golden/small_kv.npz, produced by the oracle) for the layer
    stack and the head kernels of a 2-layer bf16 model — no oracle call at run time."""
    import os
    gold = np.load(os.path.join(os.path.dirname(__file__), "golden", "small_kv.npz"))
    gm = R.Model.synthetic(R.Config(256, 640, 2, 128, 64, 2, 1500), 5, dtype="bf16")
    hidden = np.stack([gm.decode_token_from_id(t) for t in (1, 2, 3)])
    np.testing.assert_allclose(hidden, gold["hidden"], atol=2e-4, rtol=1e-4)
    tv, ti = gm.decode_token_topk_from_id(9, 4)
    np.testing.assert_array_equal(ti, gold["topk_idxs"])
    np.testing.assert_allclose(tv, gold["topk_vals"], atol=1e-3)
    mx, sm = gm.decode_token_block_stats_from_id(11, 1.25)
    np.testing.assert_allclose(mx, gold["maxes"], atol=1e-3)
    np.testing.assert_allclose(sm, gold["sums"], atol=1e-2)
    np.testing.assert_allclose(gm.materialize_current_logits_block(5), gold["block5"], atol=1e-3)
    assert gm.decode_token_argmax_from_id(7) == int(gold["argmax"])


def test_kv_cache_dtype_option(R, oracle):
    """The KV cache's storage is an option of its own: a bf16 model keeps fp16 keys and values by
    default and bf16 ones on request; each agrees with the oracle that rounds its cache the same way."""
    O = oracle
    for kv, odt in ((None, O.F16), ("bf16", O.BF16)):
        oc = oracle_cfg(O, *SMALL, dtype="bf16")
        om = O.Model.synth(oc, 5).set_kv_dtype(odt)
        gm = R.Model.synthetic(gpu_cfg(R, oc), 5, dtype="bf16", kv_dtype=kv)
        cache = O.Cache(om, kv_round=1)
        tok = 3
        for _ in range(10):
            a, b = gm.decode_token_logits_from_id(tok), cache.decode_logits(tok)
            assert np.abs(a - b).max() < tol("bf16")
            tok = int(np.argmax(b))
    with pytest.raises(R.CudaDecodeError, match="KV-cache dtype"):
        R.Model.synthetic(gpu_cfg(R, oc), 5, dtype="f32", kv_dtype="f16")


def test_a_wait_on_a_silent_peer_runs_out_and_reports(R):
    """Two ranks of a tensor-parallel model built in one process on one GPU, of which only rank 0 is
    ever driven: its wait for rank 1's partial sums is bounded (20 ms here), runs out, and the call
    returns CD_ERR_DEVICE_WAIT instead of spinning; the handle stays valid and a second call
    reports the same again (the error word is cleared between calls)."""
    import time
    cfg = R.Config(256, 640, 2, 128, 64, 2, 320)
    ranks = [R.Model.synthetic(cfg, 5, dtype="bf16", tp_rank=r, tp_world=2, wait_us=20000) for r in range(2)]
    regions = [m.tp_region_ptr() for m in ranks]
    for m in ranks:
        m.tp_connect_ptrs(regions)
    for _ in range(2):
        t0 = time.time()
        with pytest.raises(R.CudaDecodeError, match="tensor-parallel peer") as exc:
            ranks[0].decode_token_argmax_from_id(1)
        assert exc.value.code == R._ffi.ERR_DEVICE_WAIT
        assert time.time() - t0 < 5.0
        assert ranks[0].len() == 0
    with pytest.raises(R.CudaDecodeError, match="tensor-parallel peer"):
        ranks[0].decode_steps_greedy(1, 8)      # every later wait of the call returns at once: one budget, not one per all-reduce
    ranks[0].set_len(0)
    for m in ranks:
        m.close()


@pytest.mark.parametrize("dtype", ["bf16", "fp8"])
def test_a_weight_stage_that_never_arrives_runs_the_ring_wait_out(R, dtype):
    """The copy ring's bounded waits: with the test hook on (cd_options.test_flags bit 3) the first CTA of every streamed
    GEMV never requests its last stage, its consumers' wait for that stage runs out (a short limit under the hook), the
    kernel records the expiry, waits - bounded - for what is in flight and returns; the call reports CD_ERR_DEVICE_WAIT
    naming the ring, the handle stays valid (state calls work, a second token call reports the same), nothing faults."""
    import time
    cfg = R.Config(256, 640, 2, 128, 64, 2, 320)
    m = R.Model.synthetic(cfg, 5, dtype=dtype, mega=False, drop_stage=True)
    for _ in range(2):
        t0 = time.time()
        with pytest.raises(R.CudaDecodeError, match="weight ring: stage never filled") as exc:
            m.decode_token_argmax_from_id(1)
        assert exc.value.code == R._ffi.ERR_DEVICE_WAIT
        assert time.time() - t0 < 10.0
        m.set_len(0)
        assert m.len() == 0
    m.close()
    ok = R.Model.synthetic(cfg, 5, dtype=dtype, mega=False)  # the same model without the hook decodes
    assert 0 <= ok.decode_token_argmax_from_id(1) < cfg.vocab


@pytest.mark.parametrize("mega", [True, False])
def test_logits_without_a_finite_maximum_never_become_an_address(R, oracle, mega):
    """A model whose final gamma is NaN has NaN logits at every row; the device's arg-max then has no winner and its
    "no row" id must not be used as a row of the embedding table by the next step of an on-device loop: the step falls
    back to row 0, records it, and the call reports the bad id instead of reading past the table."""
    oc = oracle_cfg(oracle, 256, 640, 2, 128, 64, 2, 320, dtype="f32")
    om = oracle.Model.synth(oc, 3)
    layers = [{n: om.tensor(getattr(oracle, "T_" + n.upper()), l) for n in ("wq", "wk", "wv", "wo", "w1", "w3", "w2", "gamma1", "gamma2")}
              for l in range(oc.nlayers)]
    head = {"gamma_final": np.full(oc.dim, np.nan, dtype=np.float32), "embed": om.tensor(oracle.T_EMBED)}
    gm = R.Model.new(gpu_cfg(R, oc), layers, head, dtype="bf16", mega=mega)
    assert np.isnan(gm.decode_token_logits_from_id(1)).all()
    gm.set_len(0)
    with pytest.raises(R.CudaDecodeError, match="outside the vocabulary"):
        gm.decode_steps_greedy(1, 6)
    gm.set_len(0)
    good = R.Model.new(gpu_cfg(R, oc), layers, dict(head, gamma_final=np.ones(oc.dim, dtype=np.float32)), dtype="bf16", mega=mega)
    assert all(0 <= t < oc.vocab for t in good.decode_steps_greedy(1, 6).tolist())

GROUPED_CASES = [
    # dims (dim, hidden, heads, hd, seq, layers, vocab), kv heads, type, page tokens, cached positions
    ((2048, 4128, 16, 128, 2304, 2, 3000), 4, "bf16", 64, 2001),  # four q heads per kv head, several tiles per CTA
    ((1024, 2080, 8, 128, 1024, 2, 3000), 1, "f16", 64, 700),     # eight q heads per kv head
    ((1024, 2080, 16, 64, 512, 2, 3000), 4, "bf16", 16, 77),      # head width 64, 16-token tiles
    ((512, 1056, 8, 64, 512, 2, 3000), 1, "f16", 8, 130),         # tiles of one warp
    ((512, 1056, 4, 128, 64, 2, 3000), 1, "bf16", 64, 1),         # the first positions
]


@pytest.mark.parametrize("dims,kv_heads,dtype,page,cached", GROUPED_CASES)
def test_grouped_queries_on_the_persistent_kernel(R, dims, kv_heads, dtype, page, cached):
    """Four and eight q heads per kv head: scores on the tensor cores (q as fp16 hi + lo pairs) against the kernel per operator.
    Inputs differ by at most 2^-23 relative, sums by their order; a cache entry may round to its neighbour: 2e-4 of the logits."""
    dim, hidden, heads, hd, seq, layers, vocab = dims
    cfg = R.Config(dim, hidden, heads, hd, seq, layers, vocab, kv_heads=kv_heads)
    a, b = (R.Model.synthetic(cfg, 7, dtype=dtype, page_tokens=page, mega=mega) for mega in (True, False))
    prompt = np.random.default_rng(1).integers(0, vocab, cached).astype(np.uint32)
    for m in (a, b):
        m.prefill(prompt, want_logits=False)
    before = a.kernel_launches()
    for tok in (5, 9, 77):
        x, y = a.decode_token_logits_from_id(tok), b.decode_token_logits_from_id(tok)
        assert np.abs(x - y).max() < 2e-4 * np.abs(y).max()
    assert a.kernel_launches() - before == 6  # the persistent kernel and the position's advance


@pytest.mark.parametrize("heads,kv_heads,hd", [(37, 37, 64), (2, 2, 128), (8, 2, 64)])
@pytest.mark.parametrize("logits", [True, False])
def test_phase_stamps_of_the_persistent_kernel_fill_their_rows(R, heads, kv_heads, hd, logits):
    """Start, two stamps per phase of a layer, end: of the first and the last CTA, whether the last one has attention work
    (37 kv heads of four CTAs each) or not.  A stamp too many would land on the other row, or behind the buffer."""
    cfg = R.Config(512, 640, heads, hd, 512, 3, 1500, kv_heads=kv_heads)
    m = R.Model.synthetic(cfg, 7, dtype="bf16", trace=True, mega=True)
    m.prefill(np.arange(300, dtype=np.uint32), want_logits=False)
    m.decode_token_logits_from_id(5) if logits else m.decode_token_from_id(5)
    n = 10 * cfg.nlayers + 2
    out, count = np.zeros(2 * n, dtype=np.uint64), ctypes.c_size_t()
    from rustane_b200 import _ffi
    assert _ffi.lib.cd_debug_phase_trace(m._h, out.ctypes.data_as(ctypes.POINTER(ctypes.c_uint64)), out.size, ctypes.byref(count)) == 0
    assert count.value == 2 * n
    rows = out.reshape(2, n).astype(np.int64)
    assert (rows > 0).all() and (np.diff(rows, axis=1) >= 0).all()
    assert abs(int(rows[0, 0]) - int(rows[1, 0])) < 1_000_000  # both of the same token


@pytest.mark.parametrize("ring_kb,launches", [(80, 2), (70, None), (0, 2)])
def test_a_large_vocabulary_leaves_the_ring_its_shared_memory(R, ring_kb, launches):
    """A CTA of the persistent kernel keeps its rows' partial sums (here 888 rows of the LM head) and the residual entries of its
    few rows of the stream beside the ring.  80 KB hold both with four stages; 70 KB do not, and the token runs a kernel per
    operator.  Same logits every way (sums in another order, a cache entry may round to its neighbour: 2e-4)."""
    cfg = R.Config(256, 640, 2, 128, 64, 2, 131072)
    m = R.Model.synthetic(cfg, 7, dtype="bf16", ring_kb=ring_kb, mega=True, use_graph=True)
    ref = R.Model.synthetic(cfg, 7, dtype="bf16", mega=False)
    for t in (5, 131071, 9):
        before = m.kernel_launches()
        x, y = m.decode_token_logits_from_id(t), ref.decode_token_logits_from_id(t)
        n = m.kernel_launches() - before
        assert n == launches if launches else n > 2
        assert np.abs(x - y).max() < 2e-4 * np.abs(y).max()


@pytest.mark.parametrize("use_graph", [False, True])
def test_form_of_a_token_by_its_position(R, use_graph):
    """Eight q heads on one kv head: a few CTAs walk the cache in the persistent kernel, so tokens behind a long enough context run
    a kernel per operator.  Both forms in one sequence, either way across the line, give what one kernel per operator gives (sums
    in another order, a cache entry may round to its neighbour: 2e-4 of the logits); mega=True keeps the one kernel."""
    cfg = R.Config(1024, 3072, 8, 128, 1024, 2, 3000, kv_heads=1)
    make = lambda mega: R.Model.synthetic(cfg, 7, dtype="bf16", mega=mega, use_graph=use_graph)
    auto, always, never = make(None), make(True), make(False)
    prompt = np.random.default_rng(1).integers(0, 3000, 470).astype(np.uint32)
    for m in (auto, always, never):
        m.prefill(prompt, want_logits=False)

    def step(m, tok):
        before = m.kernel_launches()
        x = m.decode_token_logits_from_id(tok)
        return x, m.kernel_launches() - before

    one = []
    for tok in range(60):
        (x, n), (y, k), (z, _) = step(auto, tok), step(always, tok), step(never, tok)
        assert k == 2 and max(np.abs(x - z).max(), np.abs(y - z).max()) < 2e-4 * np.abs(z).max()
        one.append(n == 2)
    assert one[0] and not one[-1] and one == sorted(one, reverse=True)  # short ones as one kernel, long ones not
    line = 470 + sum(one)
    for m in (auto, never):
        m.set_len(line - 3)
    assert [step(auto, t)[1] == 2 for t in range(6)] == [True] * 3 + [False] * 3
    auto.set_len(line - 8)
    before = auto.kernel_launches()
    ids = auto.decode_steps_greedy(5, 16)
    assert auto.kernel_launches() - before == 1 + 8 * 2 + 8 * (5 * cfg.nlayers + 3)
    never.set_len(line - 8)
    assert np.array_equal(ids, never.decode_steps_greedy(5, 16))


@pytest.mark.parametrize("hidden", [12544, 13312, 13824, 16384])
def test_widest_rows_of_the_persistent_kernel(R, hidden):
    """Seven and eight chunks a thread of W2's rows: as one kernel where four ring stages fit beside the L1 that its spilled registers need, else per operator."""
    cfg = R.Config(2176, hidden, 17, 128, 64, 2, 1500)
    a, b = (R.Model.synthetic(cfg, 3, dtype="bf16", mega=mega) for mega in (None, False))
    before = a.kernel_launches()
    for t in (7, 1499, 3):
        x, y = a.decode_token_logits_from_id(t), b.decode_token_logits_from_id(t)
        assert np.abs(x - y).max() < 2e-4 * np.abs(y).max()
    assert (a.kernel_launches() - before == 6) == (hidden < 13800)


@pytest.mark.parametrize("dims,kv_heads,dtype", [((576, 1536, 8, 64, 4096, 13, 10303), 1, "bf16"), ((1664, 3328, 26, 64, 4096, 20, 300), 13, "fp8"),
                                                 ((2624, 6208, 41, 64, 4096, 16, 2778), 41, "fp8")])
def test_a_ring_that_just_fits(R, dims, kv_heads, dtype):
    """Shapes whose stages, beside the other buffers, come within 100 bytes of the shared memory a block can have."""
    cfg = R.Config(*dims, kv_heads=kv_heads)
    a, b = (R.Model.synthetic(cfg, 3, dtype=dtype, mega=mega, use_graph=True) for mega in (True, False))
    before = a.kernel_launches()
    for t in (7, 299, 3):
        x, y = a.decode_token_logits_from_id(t), b.decode_token_logits_from_id(t)
        assert np.abs(x - y).max() < 1e-3 * np.abs(y).max()  # (up to 20 layers of caches that may round to the neighbour)
    assert a.kernel_launches() - before == 6
