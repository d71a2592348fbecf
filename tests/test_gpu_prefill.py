"""The batched tensor-core prompt pass against the oracle and against the per-token path.

The batched pass rounds every GEMM input to the model's 16-bit type (as a hi + lo pair by
default), so it cannot be bit-identical to the fp32-activation oracle; the bound asserted is
the stated 2e-2 on logits, and the measured distance (a few 1e-4 on these shapes) is checked
against a tighter 2e-3.  With CD_PREFILL=fast (single rounding) the measured distance is
about 1e-2 of the logit range and only the stated bound is asserted.  What the pass leaves in
the KV pages is checked by continuing with ordinary decode steps against the oracle's cache.
"""
import os

import numpy as np
import pytest

from helpers import gpu_cfg, oracle_cfg, top2_gap

pytestmark = pytest.mark.gpu

LOGIT_TOL = 2e-2
SPLIT_TOL = 2e-3

CASES = [
    # dims (dim, hidden, heads, hd, seq, nlayers, vocab), dtype, config extras, prompt length
    ((256, 640, 2, 128, 256, 2, 320), "bf16", {}, 37),                                 # one partial 128-row tile
    ((256, 640, 2, 128, 256, 2, 320), "f16", {}, 130),                                 # two row tiles, ragged
    ((256, 512, 4, 64, 300, 2, 512), "bf16", dict(kv_heads=2, activation=1), 200),     # hd 64, GQA, LeakyReLU^2
    ((512, 1536, 8, 64, 512, 3, 8192), "bf16", dict(untied=1, page_tokens=16), 300),   # small pages, untied head
    ((1536, 4096, 12, 128, 1024, 2, 32000), "f16", {}, 512),                           # configuration-2 widths
]


@pytest.fixture(autouse=True)
def _restore_env():
    old = os.environ.get("CD_PREFILL")
    yield
    if old is None:
        os.environ.pop("CD_PREFILL", None)
    else:
        os.environ["CD_PREFILL"] = old


def _models(R, O, dims, dtype, kw):
    kw = dict(kw)
    opts = {k: kw.pop(k) for k in ("page_tokens",) if k in kw}
    oc = oracle_cfg(O, *dims, dtype=dtype, **kw)
    om = O.Model.synth(oc, 5)
    gm = R.Model.synthetic(gpu_cfg(R, oc), 5, untied_head=bool(oc.untied), dtype=dtype, activation=oc.activation, **opts)
    return oc, om, gm


def _oracle_prefill(O, om, prompt):
    cache = O.Cache(om, kv_round=1)
    for t in prompt[:-1]:
        cache.decode_token_from_id(int(t))
    return cache, cache.decode_logits(int(prompt[-1]))


@pytest.mark.parametrize("dims,dtype,kw,n", CASES)
@pytest.mark.parametrize("mode", ["split", "fast"])
def test_batched_prefill_matches_oracle(R, oracle, dims, dtype, kw, n, mode):
    oc, om, gm = _models(R, oracle, dims, dtype, kw)
    prompt = oracle.synth_prompt(7, oc.vocab, n)
    cache, ref = _oracle_prefill(oracle, om, prompt)
    os.environ["CD_PREFILL"] = mode
    launches = gm.kernel_launches()
    got = gm.prefill(prompt)
    assert gm.kernel_launches() - launches < 12 * oc.nlayers + 8     # the batched pass, not n single-token steps
    assert gm.len() == n
    err = float(np.abs(got - ref).max())
    assert err < (SPLIT_TOL if mode == "split" else LOGIT_TOL), err
    # the K / V the pass wrote: continue with ordinary decode steps
    tok, worst = int(np.argmax(ref)), 0.0
    for _ in range(6):
        a, b = gm.decode_token_logits_from_id(tok), cache.decode_logits(tok)
        worst = max(worst, float(np.abs(a - b).max()))
        tok = int(np.argmax(b))
    assert worst < (SPLIT_TOL if mode == "split" else LOGIT_TOL), worst


def test_batched_prefill_in_chunks_and_against_per_token_path(R, oracle):
    """A prompt fed as two chunks (the second attends the first through the pages) equals the
    oracle, and greedy decoding after a batched prompt pass equals decoding after the
    per-token pass when the oracle's own top-2 gap is well above the measured distance."""
    dims, dtype = (512, 1536, 8, 64, 512, 3, 8192), "bf16"
    oc, om, gm = _models(R, oracle, dims, dtype, dict(untied=1))
    prompt = oracle.synth_prompt(8, oc.vocab, 210)
    cache, ref = _oracle_prefill(oracle, om, prompt)
    os.environ["CD_PREFILL"] = "split"
    gm.prefill(prompt[:90], want_logits=False)
    got = gm.prefill(prompt[90:])
    assert gm.len() == 210
    assert float(np.abs(got - ref).max()) < SPLIT_TOL
    ids_batched = gm.decode_steps_greedy(int(np.argmax(got)), 16).tolist()
    os.environ["CD_PREFILL"] = "token"
    gm.set_len(0)
    tok_logits = gm.prefill(prompt)
    assert float(np.abs(tok_logits - ref).max()) < 1e-3
    ids_token = gm.decode_steps_greedy(int(np.argmax(tok_logits)), 16).tolist()
    ref_ids, cur = [], int(np.argmax(ref))
    for _ in range(16):
        lg = cache.decode_logits(cur)
        if top2_gap(lg) < 10 * SPLIT_TOL:
            break
        cur = int(np.argmax(lg))
        ref_ids.append(cur)
    assert len(ref_ids) >= 1, "the oracle's own first step is a near tie: pick another prompt seed"
    assert ids_token[:len(ref_ids)] == ref_ids
    assert ids_batched[:len(ref_ids)] == ref_ids


def test_short_prompts_and_fp32_models_keep_the_per_token_path(R, oracle):
    oc, om, gm = _models(R, oracle, (256, 640, 2, 128, 64, 2, 320), "f32", {})
    prompt = oracle.synth_prompt(1, oc.vocab, 40)
    cache, ref = _oracle_prefill(oracle, om, prompt)
    assert float(np.abs(gm.prefill(prompt) - ref).max()) < 1e-4     # fp32 storage: not a tensor-core case
    oc, om, gm = _models(R, oracle, (256, 640, 2, 128, 64, 2, 320), "bf16", {})
    cache, ref = _oracle_prefill(oracle, om, prompt[:5])
    assert float(np.abs(gm.prefill(prompt[:5]) - ref).max()) < 1e-3  # below the batching threshold


@pytest.mark.parametrize("dtype", ["bf16", "f32"])
def test_logits_at_chosen_places_of_a_prompt(R, oracle, dtype):
    """cd_prefill_logits on the dense family, through the batched pass (bf16) and the per-token path (f32): the logits at
    places in any order equal the oracle's, and a dense cache rewinds to any length."""
    oc, om, gm = _models(R, oracle, (256, 640, 2, 128, 64, 2, 320), dtype, {})
    prompt = oracle.synth_prompt(2, oc.vocab, 40)
    cache = oracle.Cache(om, kv_round=0 if dtype == "f32" else 1)
    ref = np.stack([cache.decode_logits(int(t)) for t in prompt])
    want = [39, 0, 17, 17]
    got = gm.prefill_logits(prompt, want)
    assert float(np.abs(got - ref[want]).max()) < (1e-4 if dtype == "f32" else SPLIT_TOL)
    assert gm.len() == 40 and gm.can_rewind(11)
    gm.set_len(11)
    assert float(np.abs(gm.prefill_logits(prompt[11:16], [4]) - ref[15]).max()) < (1e-4 if dtype == "f32" else SPLIT_TOL)
    with pytest.raises(R.CudaDecodeError):
        gm.prefill_logits(prompt[:3], [3])


@pytest.mark.parametrize("hd,kv_heads,page", [(64, 1, 32), (128, 4, 64), (128, 2, 128)])
@pytest.mark.parametrize("cached,n", [(0, 8), (0, 127), (0, 128), (0, 129), (0, 257), (100, 156), (130, 255)])
def test_attention_at_the_edges_of_its_tiles(R, oracle, hd, kv_heads, page, cached, n):
    """Prompt lengths around 128 keys and 256 query rows, with and without cached tokens ahead of the chunk, over grouped heads
    and page sizes.  Whatever the cache holds behind the last key (NaN here) must not reach the logits."""
    dims = (256, 320, 4, hd, 512, 2, 300)
    oc, om, gm = _models(R, oracle, dims, "bf16", dict(kv_heads=kv_heads, page_tokens=page))
    nan = np.full(oc.kv_heads * hd * oc.seq, np.nan, np.float32)
    for l in range(oc.nlayers):
        gm.seed_layer_cache_from_channel_first(l, oc.seq, nan, nan)
    prompt = oracle.synth_prompt(9, oc.vocab, cached + n)
    _, ref = _oracle_prefill(oracle, om, prompt)
    gm.set_len(0)
    if cached:
        gm.prefill(prompt[:cached], want_logits=False)
    assert float(np.abs(gm.prefill(prompt[cached:]) - ref).max()) < SPLIT_TOL


@pytest.mark.parametrize("mode", ["split", "fast"])
@pytest.mark.parametrize("n,hidden", [(40, 48), (128, 9616), (129, 9616), (300, 11008), (1030, 9616)])
def test_tiles_of_the_linears(R, oracle, n, hidden, mode):
    """Tiles of one CTA and of a pair, several of them in turn on one unit (both accumulators used again), with a last row tile
    of one row or of one of the pair's halves, and columns that end inside a tile."""
    oc, om, gm = _models(R, oracle, (160, hidden, 2, 64, 1100, 1, 300), "bf16", {})
    prompt = oracle.synth_prompt(11, oc.vocab, n)
    _, ref = _oracle_prefill(oracle, om, prompt)
    os.environ["CD_PREFILL"] = mode
    assert float(np.abs(gm.prefill(prompt) - ref).max()) < (SPLIT_TOL if mode == "split" else LOGIT_TOL)
