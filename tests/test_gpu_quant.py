"""Quantised linears (FP8-E4M3 per output channel, INT4 group-32) against the oracle.

The reference has no quantised path, so the rule itself is builder-defined; what is pinned is
that the CUDA library and the oracle quantise identically and that decoding with the
quantised rows equals the oracle run on the dequantised values.  Both sides then hold
the same numbers, so the stated bound is the one of the 16-bit formats: logits within 1e-3
max-abs (summation order plus one-ulp flips of bf16 KV values), greedy ids identical.
"""
import numpy as np
import pytest

from helpers import gpu_cfg, oracle_cfg, top2_gap

pytestmark = pytest.mark.gpu

QUANT_TOL = 1e-3
MODES = {"fp8": 3, "int4": 4}

SHAPES = [
    ((256, 640, 2, 128, 64, 2, 320), {}),                      # the reference's small decode shape
    ((512, 1536, 8, 64, 96, 3, 8192), dict(untied=1)),         # configuration-1 widths, untied head
    ((384, 992, 3, 128, 80, 2, 1000), dict(page_tokens=16)),   # K = 992 = 31 groups: partial chunk rows
    ((256, 512, 4, 64, 80, 2, 512), dict(kv_heads=2, activation=1)),
]


def _pair(R, O, dims, dtype, seed=9, **kw):
    opts = {k: kw.pop(k) for k in ("use_graph", "page_tokens") if k in kw}
    oc = oracle_cfg(O, *dims, dtype="f32", **kw)
    om = O.Model.synth_quant(oc, seed, MODES[dtype])
    gm = R.Model.synthetic(gpu_cfg(R, oc), seed, untied_head=bool(oc.untied), dtype=dtype, activation=oc.activation, **opts)
    return oc, om, gm


@pytest.mark.parametrize("dims,kw", SHAPES)
@pytest.mark.parametrize("dtype", ["fp8", "int4"])
def test_quantised_decode_matches_oracle_on_dequantised_weights(R, oracle, dims, kw, dtype):
    oc, om, gm = _pair(R, oracle, dims, dtype, **dict(kw))
    cache = oracle.Cache(om, kv_round=1)
    tok, worst = 3, 0.0
    for _ in range(16):
        a, b = gm.decode_token_logits_from_id(tok), cache.decode_logits(tok)
        worst = max(worst, float(np.abs(a - b).max()))
        tok = int(np.argmax(b))
    assert worst < QUANT_TOL, worst


@pytest.mark.parametrize("dtype", ["fp8", "int4"])
def test_quantised_greedy_loop_and_host_weights(R, oracle, dtype):
    """Greedy ids of the on-device loop equal the oracle's; a model built from host fp32
    tensors (relayout + quantise at construction) equals the self-generated one bit for bit."""
    dims = (512, 1536, 8, 64, 128, 4, 8192)
    oc, om, gm = _pair(R, oracle, dims, dtype, use_graph=True)
    prompt = oracle.synth_prompt(1, oc.vocab, 8)
    cache = oracle.Cache(om, kv_round=1)
    for t in prompt[:-1]:
        cache.decode_token_from_id(int(t))
    ref = cache.decode_logits(int(prompt[-1]))
    got = gm.prefill(prompt)
    assert np.abs(got - ref).max() < QUANT_TOL
    assert top2_gap(ref) > QUANT_TOL
    tok = int(np.argmax(ref))
    gpu_ids = gm.decode_steps_greedy(tok, 24).tolist()
    ref_ids, cur = [], tok
    for _ in range(24):
        cur = cache.decode_token_argmax_from_id(cur)
        ref_ids.append(cur)
    assert gpu_ids == ref_ids
    # host-tensor construction: unquantised fp32 tensors in, quantised at construction
    plain = oracle.Model.synth(oracle_cfg(oracle, *dims, dtype="f32"), 9)
    layers = [{n: plain.tensor(getattr(oracle, "T_" + n.upper()), l) for n in
               ("wq", "wk", "wv", "wo", "w1", "w3", "w2", "gamma1", "gamma2")} for l in range(oc.nlayers)]
    head = {"gamma_final": plain.tensor(oracle.T_GAMMA_FINAL), "embed": plain.tensor(oracle.T_EMBED)}
    gm2 = R.Model.new(gpu_cfg(R, oc), layers, head, dtype=dtype)
    gm3 = R.Model.synthetic(gpu_cfg(R, oc), 9, dtype=dtype)
    for t in (1, 7, 300):
        assert np.array_equal(gm2.decode_token_logits_from_id(t), gm3.decode_token_logits_from_id(t))


def test_quantised_rejections(R):
    cfg = R.Config(264, 640, 2, 128, 64, 2, 320)  # dim not a multiple of 16 / 32
    for dtype in ("fp8", "int4"):
        with pytest.raises(Exception):
            R.Model.synthetic(cfg, 1, dtype=dtype)


@pytest.mark.parametrize("dims,n", [((512, 1536, 8, 64, 256, 3, 8192), 150), ((256, 640, 2, 128, 128, 2, 320), 40)])
def test_fp8_prompt_pass_on_the_tensor_cores(R, oracle, dims, n, monkeypatch):
    """FP8 models run prompts of 8+ tokens through the tensor-core pass (e4m3 values widened exactly to
    bf16 per layer, row scales on the GEMM's output columns); INT4 models keep the per-token path.
    Same bound as the bf16 prompt pass: 2e-3 against the oracle on the dequantised weights."""
    oc, om, gm = _pair(R, oracle, dims, "fp8")
    prompt = oracle.synth_prompt(2, oc.vocab, n)
    cache = oracle.Cache(om, kv_round=1)
    for t in prompt[:-1]:
        cache.decode_token_from_id(int(t))
    ref = cache.decode_logits(int(prompt[-1]))
    launches = gm.kernel_launches()
    got = gm.prefill(prompt)
    assert gm.kernel_launches() - launches < 20 * oc.nlayers + 8      # the batched pass, not n single-token steps
    assert float(np.abs(got - ref).max()) < 2e-3
    tok = int(np.argmax(ref))
    for _ in range(4):  # the K / V it wrote, through ordinary decode steps
        a, b = gm.decode_token_logits_from_id(tok), cache.decode_logits(tok)
        assert float(np.abs(a - b).max()) < 2e-3
        tok = int(np.argmax(b))
    monkeypatch.setenv("CD_PREFILL", "token")
    gm.set_len(0)
    assert float(np.abs(gm.prefill(prompt) - ref).max()) < QUANT_TOL


def _row_bytes(dtype, k):
    return k + 16 if dtype == "fp8" else (k // 2 + k // 16 + 15) // 16 * 16


@pytest.mark.parametrize("dtype", ["fp8", "int4"])
def test_stored_quantised_checkpoint_loads_bit_identically(R, tmp_path, dtype):
    """A plain RSTK file converted once (cd_convert_checkpoint) loads, without conversion, to the very rows and logits
    that quantising the plain file at load produces; a tensor-parallel rank takes its shard of the stored rows (whole-row
    FP8 scales, its own INT4 groups) exactly as the load-time quantiser cuts it."""
    cfg = R.Config(256, 640, 4, 64, 64, 2, 320, kv_heads=2)
    plain, quant = str(tmp_path / "plain.rstk"), str(tmp_path / ("q_%s.rstk" % dtype))
    R.write_synthetic_checkpoint(plain, cfg, dtype="bf16", untied_head=True, seed=6)
    R.convert_checkpoint(plain, quant, dtype)
    info = R.checkpoint_info(quant)
    assert info["quantised_linears"] and info["untied_head"] and info["dtype"] == MODES[dtype] and info["version"] == 3
    a = R.Model.from_checkpoint(plain, dtype=dtype)   # quantised at load
    b = R.Model.from_checkpoint(quant)                # stored rows
    widths = [(cfg.q_dim, cfg.dim), (cfg.kv_dim, cfg.dim), (cfg.kv_dim, cfg.dim), (cfg.dim, cfg.q_dim),
              (cfg.hidden, cfg.dim), (cfg.hidden, cfg.dim), (cfg.dim, cfg.hidden)]
    for layer in range(cfg.nlayers):
        for which, (rows, k) in enumerate(widths):
            n = rows * _row_bytes(dtype, k)
            assert np.array_equal(a.linear_rows(layer, which, n), b.linear_rows(layer, which, n)), (layer, which)
    tok = 5
    for _ in range(6):
        la, lb = a.decode_token_logits_from_id(tok), b.decode_token_logits_from_id(tok)
        assert np.array_equal(la, lb)
        tok = int(np.argmax(la))
    with pytest.raises(R.CudaDecodeError, match="loads in its own format only"):
        R.Model.from_checkpoint(quant, dtype="bf16")
    # a live quantised model writes the same file
    again = str(tmp_path / "again.rstk")
    a.save_quantised(again)
    assert open(again, "rb").read() == open(quant, "rb").read()
    a.close(); b.close()
    # rank 1 of 2: shards of the stored rows against shards quantised at load (construction only; nothing is decoded)
    sa = R.Model.from_checkpoint(plain, dtype=dtype, tp_rank=1, tp_world=2)
    sb = R.Model.from_checkpoint(quant, tp_rank=1, tp_world=2)
    half = [(cfg.q_dim // 2, cfg.dim), (cfg.kv_dim // 2, cfg.dim), (cfg.kv_dim // 2, cfg.dim), (cfg.dim, cfg.q_dim // 2),
            (cfg.hidden // 2, cfg.dim), (cfg.hidden // 2, cfg.dim), (cfg.dim, cfg.hidden // 2)]
    for which, (rows, k) in enumerate(half):
        n = rows * _row_bytes(dtype, k)
        assert np.array_equal(sa.linear_rows(1, which, n), sb.linear_rows(1, which, n)), which
    sa.close(); sb.close()


@pytest.mark.parametrize("dim,hidden,heads,hd,seq", [(256, 640, 4, 64, 64), (1024, 2832, 8, 128, 256), (512, 8208, 4, 128, 64), (4096 + 128, 8192, 33, 128, 64)])
def test_fp8_persistent_kernel_matches_the_kernel_per_operator(R, dim, hidden, heads, hd, seq):
    """FP8 rows through the tensor cores (fp16 weights, inputs as hi + lo pairs, fp32 sums) against the same rows through fp32
    FMAs: one to four chunks per thread, a ragged last chunk, rows that end inside a stage.  Inputs differ by at most 2^-23 relative and
    sums by their order: a few 1e-6 of logits of order one over two layers; an fp16 cache entry may round to its neighbour."""
    cfg = R.Config(dim, hidden, heads, hd, seq, 2, 1500)
    a, b = R.Model.synthetic(cfg, 3, dtype="fp8"), R.Model.synthetic(cfg, 3, dtype="fp8", mega=False)
    before = a.kernel_launches()
    for t in (7, 1499, 3, 3, 900):
        x, y = a.decode_token_logits_from_id(t), b.decode_token_logits_from_id(t)
        assert np.abs(x - y).max() < 2e-4 * np.abs(y).max()
    assert a.kernel_launches() - before == 10  # the persistent kernel and the position's advance


@pytest.mark.parametrize("value", [0.0, 1e-36, 1e-20])
@pytest.mark.parametrize("zero_gamma", [False, True])
def test_fp8_zero_and_tiny_inputs(R, value, zero_gamma):
    """A token whose embedding row is zero or tiny (padding rows of checkpoints), a zero hidden vector, a norm with a zero gamma:
    the scale that brings an input to fp16's range must not overflow, and nothing may reach the cache that disturbs later tokens."""
    cfg, rng = R.Config(256, 640, 2, 128, 64, 2, 320), np.random.default_rng(4)
    shapes = dict(wq=(256, 256), wk=(256, 256), wv=(256, 256), wo=(256, 256), w1=(256, 640), w3=(256, 640), w2=(256, 640))
    layers = [dict({n: rng.normal(0, 0.05, s).astype(np.float32) for n, s in shapes.items()}, gamma1=np.ones(256), gamma2=np.ones(256)) for _ in range(2)]
    if zero_gamma:
        layers[1]["gamma1"] = np.zeros(256)
    embed = rng.normal(0, 0.05, (320, 256)).astype(np.float32)
    embed[5] = value
    a, b = (R.Model.new(cfg, layers, dict(gamma_final=np.ones(256), embed=embed), dtype="fp8", mega=mega) for mega in (True, False))
    for t in (5, 7, 5, 9, 300):
        x, y = a.decode_token_logits_from_id(t), b.decode_token_logits_from_id(t)
        assert np.isfinite(y).all() and np.abs(x - y).max() <= 2e-4 * np.abs(y).max(), t
    x, y = a.decode_token(np.full(256, value)), b.decode_token(np.full(256, value))
    assert np.abs(x - y).max() <= 2e-4 * np.abs(y).max()
    x, y = a.decode_token_logits_from_id(11), b.decode_token_logits_from_id(11)
    assert np.abs(x - y).max() <= 2e-4 * np.abs(y).max()


@pytest.mark.parametrize("dim,hidden,vocab", [(1024, 4112, 1500), (512, 12304, 1500), (512, 16384, 1500), (4224, 15360, 1500), (512, 16384, 60000)])
def test_fp8_chunks_per_thread(R, dim, hidden, vocab):
    """The tilings of FP8 rows that the shapes above leave out: two, and four chunks a thread of W2's rows (all live at 16384).
    Beside the sums of 60000 rows of the LM head a ring of four such stages does not fit: a kernel per operator."""
    cfg = R.Config(dim, hidden, dim // 128, 128, 64, 2, vocab)
    a, b = R.Model.synthetic(cfg, 3, dtype="fp8", mega=True), R.Model.synthetic(cfg, 3, dtype="fp8", mega=False)
    before = a.kernel_launches()
    for t in (7, 1499, 3):
        x, y = a.decode_token_logits_from_id(t), b.decode_token_logits_from_id(t)
        assert np.abs(x - y).max() < 2e-4 * np.abs(y).max()
    assert (a.kernel_launches() - before == 6) == (vocab < 60000)


@pytest.mark.parametrize("dim,hidden,heads,kv_heads,hd,value", [
    (256, 640, 4, 4, 64, 0.0),              # one octet of groups, fewer than the warps
    (1024, 2848, 8, 8, 128, 1e-20),         # a ragged last octet
    (4096, 4128, 32, 32, 128, 1e-36),       # two chunks of W2's rows
    (512, 8224, 4, 1, 128, None),           # three, grouped heads
    (512, 12320, 4, 4, 128, None),          # four
    (4224, 15360, 33, 33, 128, None),       # two of the others' rows
    (1056, 2112, 8, 1, 64, None),           # eight q heads on one kv head
])
def test_int4_persistent_kernel_matches_the_kernel_per_operator(R, dim, hidden, heads, kv_heads, hd, value):
    """INT4 rows through the tensor cores (exact fp16 weights, inputs as hi + lo pairs, a group's sum times its scale in fp32)
    against the same rows through fp32 FMAs.  Inputs differ by at most 2^-23 relative and sums by their order: a few 1e-6 of logits
    of order one over two layers; an fp16 cache entry may round to its neighbour.  A zero or tiny input must stay finite."""
    cfg = R.Config(dim, hidden, heads, hd, 64, 2, 1500, kv_heads=kv_heads)
    a, b = (R.Model.synthetic(cfg, 3, dtype="int4", mega=mega) for mega in (True, False))
    before = a.kernel_launches()
    for t in (7, 1499, 3):
        x, y = a.decode_token_logits_from_id(t), b.decode_token_logits_from_id(t)
        assert np.abs(x - y).max() < 2e-4 * np.abs(y).max()
    assert a.kernel_launches() - before == 6
    if value is not None:
        x, y = a.decode_token(np.full(dim, value)), b.decode_token(np.full(dim, value))
        assert np.isfinite(y).all() and np.abs(x - y).max() <= 2e-4 * np.abs(y).max()
        x, y = a.decode_token_logits_from_id(900), b.decode_token_logits_from_id(900)
        assert np.abs(x - y).max() < 2e-4 * np.abs(y).max()


@pytest.mark.parametrize("dtype,limit", [("int4", 3e-6), ("fp8", 3e-6)])
@pytest.mark.parametrize("dim,hidden", [(256, 640), (512, 1536), (1024, 2848), (512, 12320)])
def test_quantised_rows_on_the_tensor_cores_keep_the_inputs_23_bits(R, dim, hidden, dtype, limit):
    """One layer's FFN alone (W_v = 0: no rounded cache entry on the way), rows through the tensor cores and through fp32 FMAs, on
    inputs whose largest is some hundred times the typical one.  Input pairs are off by 2^-23 and sums of K products round at 2^-24 of
    their terms: below 1e-6 of the output's norm.  Nibbles as fp16 subnormals had 3e-5 (an MMA aligns its products as if the leading
    zeros of a subnormal were digits), inputs without their lo parts 1e-4."""
    rng = np.random.default_rng(dim + hidden)
    mat = lambda *s: (rng.standard_normal(s) / 25.0).astype(np.float32)  # noqa: E731
    heads, hd = dim // 64, 64
    L = dict(wq=mat(dim, dim), wk=mat(dim, dim), wv=np.zeros((dim, dim), np.float32), wo=mat(dim, dim), w1=mat(dim, hidden), w3=mat(dim, hidden), w2=mat(dim, hidden),
             gamma1=np.ones(dim, np.float32), gamma2=np.ones(dim, np.float32))
    head = dict(gamma_final=np.ones(dim, np.float32), embed=mat(300, dim))
    cfg = R.Config(dim, hidden, heads, hd, 64, 1, 300)
    a, b = (R.Model.new(cfg, [L], head, dtype=dtype, mega=mega) for mega in (True, False))
    worst = 0.0
    for _ in range(6):
        x = (rng.standard_normal(dim) * np.exp(1.5 * rng.standard_normal(dim))).astype(np.float32)
        outs = []
        for m in (a, b):
            m.set_len(0)
            before = m.kernel_launches()
            outs.append(m.decode_token(x).astype(np.float64) - x)
            if m is a:
                assert m.kernel_launches() - before <= 2  # the persistent kernel
        worst = max(worst, np.linalg.norm(outs[0] - outs[1]) / np.linalg.norm(outs[1]))
    assert worst < limit, worst
