"""Products of a few rows over row-tiled weights (the mma.sync GEMM): decode batches and short prompts."""
import numpy as np
import pytest

import adam_b200 as A
from adam_b200 import gguf_blocks as gb
from oracle import q4_blocks

from tests.test_gpu_gemv import _gemv

pytestmark = pytest.mark.gpu


def _error(gpu, ggml_type, raw, N, K, x, policy):
    gpu.tc_gemm_policy(policy)
    try:
        y = _gemv(gpu, ggml_type, raw, N, K, x, tile=True).astype(np.float64)
    finally:
        gpu.tc_gemm_policy(1)
    ref = x.astype(np.float64) @ q4_blocks.dequant(raw.reshape(-1), ggml_type, N, K).astype(np.float64).T
    return np.linalg.norm(y - ref, axis=1) / np.linalg.norm(ref, axis=1)


# Rows around the groups of four the kernel is built for; one row group and many; K of one tile pair, of a partial last
# stage, and long; items shared between CTAs.
@pytest.mark.parametrize("mean", [0.0, 1.0])
@pytest.mark.parametrize("ggml_type,N,K,B", [
    (2, 16, 64, 5), (2, 1152, 1152, 6), (2, 1536, 1152, 8), (2, 1152, 6912, 8), (2, 2400, 320, 7), (2, 1152, 1024, 5), (2, 4624, 4160, 13), (2, 16400, 1152, 15),
    (2, 30720, 1152, 3), (12, 16, 256, 7), (12, 5392, 5376, 3), (12, 5376, 5632, 4), (12, 512, 5376, 5), (12, 5376, 1280, 8), (12, 1152, 21504, 9), (12, 5376, 21504, 12), (12, 21504, 1024, 16)])
def test_few_rows(gpu, ggml_type, N, K, B, mean):
    """Every row within 5e-7 of the exact product: 22 bits of every activation (2^-23 each, less in a sum), two additions of the
    tensor core per block rounded towards zero (2^-23 of the block's sum each), fp32 sums over the blocks; and with
    activations that have a mean within 16 of its units, for the blocks' offsets cancel what the codes' mean adds."""
    rng = np.random.default_rng(N + K + B)
    raw = {2: gb.random_q4_0_blocks, 12: gb.random_q4_k_blocks}[ggml_type](rng, N, K)
    x = (rng.standard_normal((B, K), dtype=np.float32) + np.float32(mean)) * rng.uniform(0.01, 100.0, (B, 1)).astype(np.float32)
    before = gpu.gemm_counts()
    e = _error(gpu, ggml_type, raw, N, K, x, 1)
    assert gpu.gemm_counts()["few"] == before["few"] + 1
    print(f"error {e.max():.2e}, GEMV {_error(gpu, ggml_type, raw, N, K, x, 0).max():.2e}")
    assert e.max() < 5e-7 and gpu.device_error() == 0


@pytest.mark.parametrize("ggml_type,N,K,B,few", [(2, 2560, 10240, 8, True), (2, 2560, 10240, 12, False), (12, 2560, 10240, 9, False), (2, 3072, 12288, 12, True), (2, 3072, 12288, 13, False),
                                                  (12, 1536, 14336, 16, False), (2, 4096, 14336, 16, True), (12, 21504, 5376, 16, True)])
def test_long_products_of_few_row_groups(gpu, ggml_type, N, K, B, few):
    """From 9 rows on the tcgen05 GEMM keeps products whose row groups leave SMs idle here; error as in test_few_rows and test_gemm_tiles."""
    rng = np.random.default_rng(N + K + B)
    raw = {2: gb.random_q4_0_blocks, 12: gb.random_q4_k_blocks}[ggml_type](rng, N, K)
    x = rng.standard_normal((B, K), dtype=np.float32)
    before = gpu.gemm_counts()
    e = _error(gpu, ggml_type, raw, N, K, x, 1)
    after = gpu.gemm_counts()
    assert after["few"] == before["few"] + few and after["tile_16"] == before["tile_16"] + (not few)
    assert e.max() < (5e-7 if few else 5e-6) and gpu.device_error() == 0


def _model(gpu, cfg, batch, policy, prompts, ggml_type=gb.GGML_TYPE_Q4_0):
    from adam_b200 import synth
    from adam_b200.config import GenerationConfig
    from adam_b200.engine import ADAMEngine
    gpu.tc_gemm_policy(policy)
    eng = ADAMEngine(gpu, cfg, synth.build_model(cfg, ggml_type, seed=71), kv_cap=len(prompts[0]) + 40, kv_dtype="f32", max_batch=batch)
    try:
        ids, _ = eng.generate_batch(prompts, GenerationConfig(max_tokens=4, eos_token_ids=(), temperature=0.0, top_k=1, repeat_penalty=1.0))
        eng.begin(prompts, [len(prompts[0]) + 30] * batch)
        eng.prefill(len(prompts[0]) - 1)
        eng.step(1, lm_head=True, logits=True, direct=True)
        return ids, np.stack([eng.read_logits(b) for b in range(batch)])
    finally:
        eng.close()
        gpu.tc_gemm_policy(1)


@pytest.mark.parametrize("batch", [5, 8])
def test_steps_of_a_few_sequences(gpu, batch):
    """Gate / up products, the LM head's arg-max and its stored logits against the same steps on the GEMV kernels: a dozen
    products in a row, each within 7e-7 of the exact one on either path."""
    from adam_b200 import synth
    from adam_b200.config import tiny_gemma3
    cfg = tiny_gemma3(n_layer=2, n_vocab=1008)
    prompts = [synth.random_prompt(cfg.n_vocab, 9, seed=200 + i) for i in range(batch)]
    before = gpu.gemm_counts()
    ids, logits = _model(gpu, cfg, batch, 1, prompts)
    assert gpu.gemm_counts()["few"] > before["few"]
    want_ids, want = _model(gpu, cfg, batch, 0, prompts)
    assert ids == want_ids and np.linalg.norm(logits - want) < 1e-5 * np.linalg.norm(want) and gpu.device_error() == 0


# Feed-forward blocks whose gate / up items have 18 row groups and are shared between CTAs (test_few_rows_shapes.py).
@pytest.mark.parametrize("ggml_type,n_embd,n_ff,batch", [(12, 3584, 28672, 12), (2, 3584, 28928, 16)])
def test_steps_whose_gate_up_items_are_shared(gpu, ggml_type, n_embd, n_ff, batch):
    """Against the same steps on the GEMV kernels: a dozen products in a row, each within 7e-7 of the exact one on either path."""
    from adam_b200 import synth
    from adam_b200.config import tiny_gemma3
    cfg = tiny_gemma3(n_layer=1, n_embd=n_embd, n_ff=n_ff, n_vocab=256)
    prompts = [synth.random_prompt(cfg.n_vocab, 3, seed=400 + i) for i in range(batch)]
    before = gpu.gemm_counts()
    ids, logits = _model(gpu, cfg, batch, 1, prompts, ggml_type)
    assert gpu.gemm_counts()["few_shared"] > before["few_shared"]
    want_ids, want = _model(gpu, cfg, batch, 0, prompts, ggml_type)
    assert np.linalg.norm(logits - want) < 1e-5 * np.linalg.norm(want) and ids == want_ids and gpu.device_error() == 0


@pytest.mark.parametrize("n_embd,n_ff,tokens,shared", [(256, 9472, 257, False), (2560, 10240, 513, True)])
def test_prompt_whose_gate_up_tiles_have_256_rows(gpu, n_embd, n_ff, tokens, shared):
    """512 prompt rows on a feed-forward block of 148 gate / up tiles, 1024 on one of 640 that CTAs share, against the same prompts
    on the GEMV kernels."""
    from adam_b200 import synth
    from adam_b200.config import tiny_gemma3
    cfg = tiny_gemma3(n_layer=1 if shared else 2, n_embd=n_embd, n_vocab=1008, n_ff=n_ff)
    prompts = [synth.random_prompt(cfg.n_vocab, tokens, seed=300 + i) for i in range(2)]
    before = gpu.gemm_counts()
    ids, logits = _model(gpu, cfg, 2, 1, prompts)
    after = gpu.gemm_counts()
    assert after["tile_256"] > before["tile_256"] and (after["shared"] > before["shared"] or not shared)
    want_ids, want = _model(gpu, cfg, 2, 0, prompts)
    assert ids == want_ids and np.linalg.norm(logits - want) < 1e-5 * np.linalg.norm(want) and gpu.device_error() == 0


# Gate / up products and heads of one to four groups of four rows: units of many row groups, items shared between CTAs (the pairs of
# 7168 x 4864), a last item with fewer row groups than the others.
@pytest.mark.parametrize("ggml_type,n_embd,n_ff,n_vocab,batch", [
    (12, 4864, 7168, 8208, 3), (12, 4864, 7168, 8208, 4), (12, 4864, 7168, 8208, 9), (12, 4864, 7168, 8208, 15), (2, 1152, 6912, 40016, 5), (2, 1152, 6976, 40016, 8), (2, 256, 512, 65552, 7)])
def test_steps_of_wide_blocks(gpu, ggml_type, n_embd, n_ff, n_vocab, batch):
    """Gate / up products, the arg-max and the stored logits of the few-row kernel against the GEMV kernels', as above."""
    from adam_b200 import synth
    from adam_b200.config import tiny_gemma3
    cfg = tiny_gemma3(n_layer=1, n_embd=n_embd, n_ff=n_ff, n_vocab=n_vocab)
    prompts = [synth.random_prompt(cfg.n_vocab, 2, seed=500 + i) for i in range(batch)]
    before = gpu.gemm_counts()
    ids, logits = _model(gpu, cfg, batch, 1, prompts, ggml_type)
    assert gpu.gemm_counts()["few"] >= before["few"] + 3
    want_ids, want = _model(gpu, cfg, batch, 0, prompts, ggml_type)
    assert ids == want_ids and np.linalg.norm(logits - want) < 1e-5 * np.linalg.norm(want) and gpu.device_error() == 0


@pytest.mark.parametrize("ggml_type,N,K,B", [(2, 1152, 1152, 6), (12, 5376, 5632, 4), (12, 21504, 1024, 16)])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_rows_that_are_not_finite(gpu, ggml_type, N, K, B, bad):
    """A row with an infinity or a NaN has no finite result, and the other rows have the bits that they have without it."""
    rng = np.random.default_rng(N + B)
    raw = {2: gb.random_q4_0_blocks, 12: gb.random_q4_k_blocks}[ggml_type](rng, N, K)
    x = rng.standard_normal((B, K), dtype=np.float32)
    want = _gemv(gpu, ggml_type, raw, N, K, x, tile=True)
    x[B // 2, K - 5] = bad
    before = gpu.gemm_counts()
    y = _gemv(gpu, ggml_type, raw, N, K, x, tile=True)
    assert gpu.gemm_counts()["few"] == before["few"] + 1
    others = np.arange(B) != B // 2
    assert np.array_equal(y[others], want[others]) and not np.isfinite(y[B // 2]).any()


def test_wide_weights_while_the_policy_changes(gpu):
    """Weights beyond fp16 take the few-row kernel or the GEMV, never the tcgen05 GEMM, whenever another thread sets the policy."""
    import threading
    N, K, B, calls = 64, 512, 8, 200
    rng = np.random.default_rng(5)
    raw = gb.random_q4_0_blocks(rng, N, K).copy()
    raw.reshape(-1, 18)[7::9, 0:2] = np.array([65504.0], np.float16).view(np.uint8)
    x = rng.standard_normal((B, K), dtype=np.float32)
    ref = x.astype(np.float64) @ q4_blocks.dequant(raw.reshape(-1), 2, N, K).astype(np.float64).T
    gpu.map_create_typed(81, A.DTYPE_GGUF_Q4_0, 1, N * K)
    gpu.upload_gguf_blocks(81, 2, 0, raw)
    gpu.tile_tensor(81, 0, N, K)
    gpu.map_create_typed(80, A.DTYPE_F32, 1, B * K + calls * B * N)
    gpu.scatter_contiguous(80, 0, x)
    zero = gpu.upload_dev(np.array([0], np.uint32))[0]
    outs = [gpu.upload_dev(np.array([B * K + i * B * N], np.uint32))[0] for i in range(calls)]
    done = threading.Event()

    def change():
        while not done.is_set():
            gpu.tc_gemm_policy(2)
            gpu.tc_gemm_policy(1)

    thread = threading.Thread(target=change)
    thread.start()
    try:
        for _ in range(20):
            for h in outs:
                gpu.map_matmul_t_xq4_dev(80, 81, zero, zero, h, B, K, N)
            y = gpu.gather(80, np.arange(B * K, B * K + calls * B * N, dtype=np.uint32)).view(np.float32).reshape(calls, B, N).astype(np.float64)
            assert (np.linalg.norm(y - ref, axis=(1, 2)) < 1e-6 * np.linalg.norm(ref)).all()
    finally:
        done.set()
        thread.join()
        gpu.tc_gemm_policy(1)
        for h in [zero] + outs:
            gpu.free_handle(h)
        gpu.map_destroy(80)
        gpu.map_destroy(81)
    assert gpu.device_error() == 0
