"""The kernels of a decode step at the edges of the rules that choose them; a test says which kernel it is about and sees that it ran."""
import numpy as np
import pytest

from adam_b200 import gguf_blocks as gb
from adam_b200 import synth
from adam_b200.config import GenerationConfig, tiny_gemma3
from adam_b200.engine import ADAMEngine
from oracle.decoder import OracleDecoder, dequant_model

pytestmark = pytest.mark.gpu


def _ran(gpu, before):
    return {k: n - before[k] for k, n in gpu.step_kernel_counts().items() if n > before[k]}


def _model(ggml_type=2, seed=0, **kw):
    kw = dict(dict(n_layer=2, n_embd=128, n_head=2, n_head_kv=1, head_dim=128, n_ff=128, n_vocab=256, sliding_window=0), **kw)
    act, post = kw.pop("act", "gelu"), kw.pop("post_norms", True)
    cfg = tiny_gemma3(**kw)
    cfg.ffn_act = act
    return cfg, synth.build_model(cfg, ggml_type, seed=seed, post_norms=post)


# ---- products behind the norm chain, gate / up pairs -------------------------------------------------------------------

# One row: a slice of one tile pair, ten slices and 32, the last of one pair; rows that are streamed, in uneven slices and the longest.
# Two to four: one row group per CTA and three with a CTA that is not full, 16 slices.  Kernels per layer.
@pytest.mark.parametrize("ggml_type,n_embd,n_ff,batch,act,post_norms,kernels", [
    (2, 192, 320, 1, "gelu", True, {"row": 4}), (2, 1216, 640, 1, "silu", True, {"row": 4}), (2, 4032, 192, 1, "gelu", False, {"row": 4}),
    (12, 1280, 768, 1, "silu", False, {"row": 4}), (12, 3840, 256, 1, "gelu", True, {"row": 4}),
    (2, 4160, 384, 1, "gelu", True, {"row": 2, "ring": 2}), (2, 6144, 320, 1, "silu", False, {"row": 2, "ring": 2}),
    (12, 4352, 512, 1, "gelu", True, {"row": 2, "ring": 2}),
    (2, 192, 320, 2, "gelu", True, {"rows": 4}), (2, 1152, 7040, 3, "gelu", True, {"rows": 4}), (2, 1216, 640, 4, "silu", False, {"rows": 4}),
    (2, 2048, 384, 2, "silu", True, {"rows": 4}), (12, 1280, 3328, 4, "gelu", True, {"rows": 4}), (12, 1536, 512, 3, "gelu", False, {"rows": 4})])
def test_products_of_a_step(gpu, ggml_type, n_embd, n_ff, batch, act, post_norms, kernels):
    """Logits of five steps against the oracle's: fp32 sums on both sides, in different orders."""
    cfg, tensors = _model(ggml_type, seed=n_embd, n_embd=n_embd, n_ff=n_ff, act=act, post_norms=post_norms)
    f32 = dequant_model(tensors)
    prompts = [synth.random_prompt(cfg.n_vocab, 5, seed=b) for b in range(batch)]
    eng = ADAMEngine(gpu, cfg, tensors, kv_cap=16, kv_dtype="f32", max_batch=batch)
    try:
        eng.begin(prompts, [8] * batch)
        oracles = [OracleDecoder(cfg, f32, kv_cap=16) for _ in prompts]
        for i in range(5):
            before = gpu.step_kernel_counts()
            eng.step(1, lm_head=True, logits=True, direct=True)
            ran = _ran(gpu, before)
            assert {k: ran.get(k, 0) for k in ("row", "ring", "rows")} == {k: cfg.n_layer * kernels.get(k, 0) for k in ("row", "ring", "rows")}
            for b, p in enumerate(prompts):
                want = oracles[b].forward(int(p[i]), i)
                assert np.abs(eng.read_logits(b) - want).max() <= 2e-5 * np.abs(want).max()
        assert gpu.device_error() == 0
    finally:
        eng.close()


@pytest.mark.parametrize("batch", [1, 3, 8])
def test_rows_whose_squares_overflow(gpu, batch):
    """x / sqrt(inf) is 0 for finite x, in every kernel that norms its input."""
    cfg, tensors = _model(seed=3, n_layer=1)
    tensors["blk.0.post_attention_norm.weight"] *= np.float32(1e25)
    eng = ADAMEngine(gpu, cfg, tensors, kv_cap=16, kv_dtype="f32", max_batch=batch)
    try:
        eng.begin([[7]] * batch, [4] * batch)
        with np.errstate(over="ignore"):
            want = OracleDecoder(cfg, dequant_model(tensors), kv_cap=16).forward(7, 0)
        eng.step(1, lm_head=True, logits=True, direct=True)
        for b in range(batch):
            assert np.array_equal(eng.read_logits(b), want)
    finally:
        eng.close()


# ---- attention ---------------------------------------------------------------------------------------------------------

# Heads per CTA 1, 2, 4, 8 and the odd groups; clusters of 2, 4 and 8 whose CTAs have more chunks than slots (16, 12 and fewer of them),
# splits; a window, pages that chunks of eight do not divide.
@pytest.mark.parametrize("head_dim,n_head,n_kv,window,page,batch,length,kv_dtype,kernel", [
    (256, 4, 1, 0, 64, 60, 300, "f16", "attn_cluster_2"), (256, 4, 1, 0, 64, 64, 300, "f32", "attn_cluster_2"),
    (128, 8, 1, 100, 16, 56, 260, "f16", "attn_cluster_2"), (128, 4, 4, 60, 12, 14, 420, "f32", "attn_cluster_2"),
    (256, 4, 1, 0, 64, 20, 1100, "f16", "attn_cluster_4"), (256, 4, 1, 0, 64, 17, 700, "f32", "attn_cluster_4"),
    (64, 4, 2, 0, 12, 10, 500, "f32", "attn_cluster_4"), (256, 8, 1, 0, 64, 24, 700, "f32", "attn_cluster_4"),
    (256, 4, 1, 0, 64, 12, 1100, "f32", "attn_cluster_8"), (256, 1, 1, 0, 64, 1, 2000, "f32", "attn_cluster_8"),
    (128, 2, 1, 300, 20, 5, 1000, "f16", "attn_cluster_8"), (256, 8, 2, 0, 64, 5, 1100, "f32", "attn_cluster_8"),
    (256, 4, 1, 0, 64, 40, 300, "f16", "attn_splits"), (256, 4, 1, 0, 64, 70, 200, "f32", "attn_splits"),
    (256, 5, 1, 0, 64, 20, 90, "f32", "attn_cluster_4"), (256, 6, 1, 0, 64, 20, 90, "f32", "attn_cluster_4"),
    (32, 3, 1, 0, 64, 6, 200, "f32", "attn_cluster_4"), (64, 5, 1, 0, 64, 5, 90, "f16", "attn_cluster_4"),
    (32, 6, 2, 0, 64, 4, 150, "f32", "attn_cluster_4"), (128, 7, 1, 0, 64, 2, 200, "f32", "attn_cluster_8")])
def test_attention_of_a_step(gpu, head_dim, n_head, n_kv, window, page, batch, length, kv_dtype, kernel):
    """The logits of a step behind prompts are those of the prompt kernels.  f32 cache: 2e-5 (both sides sum in fp32, in different
    orders); f16: a last-bit difference can move a cached value by one f16 step."""
    cfg, tensors = _model(seed=length, n_head=n_head, n_head_kv=n_kv, head_dim=head_dim, sliding_window=window)
    prompts = [synth.random_prompt(cfg.n_vocab, max(2, length - 3 * b), seed=70 + b) for b in range(batch)]
    eng = ADAMEngine(gpu, cfg, tensors, kv_cap=length + 8, kv_dtype=kv_dtype, max_batch=batch, window=window > 0, page_size=page)
    try:
        eng.begin(prompts, [len(p) + 2 for p in prompts])
        eng.prefill_prompts(prompts, 0)
        before = gpu.step_kernel_counts()
        eng.step(1, lm_head=True, logits=True, direct=True)
        assert {k: n for k, n in _ran(gpu, before).items() if k.startswith("attn")} == {kernel: cfg.n_layer}
        got = {b: eng.read_logits(b) for b in sorted({0, 1 % batch, batch // 3, batch // 2, batch - 1})}
        for b, g in got.items():
            want = eng.logits_trace(prompts[b])[-1]
            assert np.abs(g - want).max() <= (1e-3 if kv_dtype == "f16" else 2e-5) * np.abs(want).max(), b
        assert gpu.device_error() == 0
    finally:
        eng.close()


def _overflowing(n_layer):
    """A model whose token 5 has values in the first layer that fp16 does not hold, and whose other tokens do not: dimension 0 is
    nothing in their embeddings."""
    cfg, tensors = _model(seed=9, n_layer=n_layer)
    raw = tensors["token_embd.weight"].raw.reshape(cfg.n_vocab, -1, gb.Q4_0_BYTES)
    raw[:, 0, 2] = (raw[:, 0, 2] & 0xF0) | 8                    # the code of weight 0: zero
    raw[5, 0, 2] = (raw[5, 0, 2] & 0xF0) | 15
    tensors["blk.0.attn_norm.weight"][0] = 1e9
    return cfg, tensors


@pytest.mark.parametrize("single_launch", [False, True])
def test_pages_of_a_sequence_that_was_not_finite(gpu, single_launch):
    """What an earlier sequence left behind the newest position does not count."""
    cfg, tensors = _overflowing(2)
    toks = synth.random_prompt(cfg.n_vocab, 70, seed=1)
    toks[toks == 5] = 6
    outs = []
    for first in ([], [5] * 80):
        eng = ADAMEngine(gpu, cfg, tensors, kv_cap=96, kv_dtype="f16", single_launch=single_launch)
        try:
            if first:
                eng.begin([first], [len(first)])
                eng.step(len(first), lm_head=False)
            outs.append(eng.logits_trace(toks, by_steps=True))
        finally:
            eng.close()
    assert np.isfinite(outs[0]).all() and np.array_equal(outs[0], outs[1])


# One split, a cluster's two splits, the independent splits of many sequences.
@pytest.mark.parametrize("before,batch", [(3, 1), (150, 1), (150, 40)])
def test_values_beyond_fp16_are_infinite(gpu, before, batch):
    """The newest position's value row holds infinities: so does the attention's output, there and with their signs."""
    cfg, tensors = _overflowing(1)
    toks = synth.random_prompt(cfg.n_vocab, before, seed=2)
    toks[toks == 5] = 6
    prompt = list(toks) + [5]
    eng = ADAMEngine(gpu, cfg, tensors, kv_cap=256, kv_dtype="f16", max_batch=batch)
    try:
        eng.begin([prompt] * batch, [len(prompt) + 1] * batch)
        eng.step(before, lm_head=False, direct=True)
        eng.step(1, lm_head=False, direct=True)
        q_dim, hd = cfg.n_head * cfg.head_dim, cfg.head_dim
        for b in {0, batch - 1}:
            v = eng.read_buffer(2, q_dim + 2 * hd, b)[q_dim + hd:]
            want = np.where(np.abs(v) >= 65520.0, np.copysign(np.inf, v), 0.0)
            got = eng.read_buffer(4, q_dim, b).reshape(cfg.n_head, hd)
            assert np.isinf(want).any() and not np.isnan(got).any()
            for h in got:
                assert np.array_equal(np.where(np.isinf(h), h, 0.0), want)
    finally:
        eng.close()


# ---- sampling ----------------------------------------------------------------------------------------------------------

def test_sampling_over_a_very_large_vocabulary(gpu):
    """More groups of candidates than shared memory has room for the heads of."""
    V, hot = 37_400_000, 37_399_999
    cfg, tensors = _model(seed=4, n_layer=1, n_embd=64, n_ff=64, head_dim=32, n_vocab=64)
    small = tensors["token_embd.weight"].raw.reshape(64, -1)
    raw = np.zeros((V, small.shape[1]), np.uint8)
    raw[:8], raw[hot] = small[:8], small[8]
    tensors["token_embd.weight"] = synth.QTensor(2, V, 64, raw.reshape(-1))
    cfg.n_vocab = V
    eng = ADAMEngine(gpu, cfg, tensors, kv_cap=16, kv_dtype="f32")
    try:
        rule = dict(max_tokens=1, eos_token_ids=(), repeat_penalty=1.0)
        for prompt in ([1], [hot], [3, hot]):
            best, _ = eng.generate(prompt, GenerationConfig(top_k=1, temperature=0.0, **rule))
            drawn, stats = eng.generate(prompt, GenerationConfig(top_k=40, top_p=0.95, temperature=1e-4, seed=1, **rule))
            assert stats["sampling_mode"] == "gpu_fused_topk" and drawn == best
    finally:
        eng.close()
