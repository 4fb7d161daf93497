"""Calls of many rows at the sizes where their kernels change tiles: the tcgen05 GEMM, the LM head's arg-max on it, the
attention of prompt chunks, scoring a text, and the host side of large results."""
import gc
from dataclasses import replace

import numpy as np
import pytest

import adam_b200 as A
from adam_b200 import gguf_blocks as gb
from adam_b200 import synth
from adam_b200.config import GenerationConfig, tiny_gemma3
from adam_b200.engine import ADAMEngine
from oracle import q4_blocks
from oracle.decoder import OracleDecoder, dequant_model

from tests.test_gpu_blocks8 import _matmul
from tests.test_gpu_decoder import GREEDY
from tests.test_gpu_gemv import _gemv

pytestmark = pytest.mark.gpu


# Rows around the tiles of 16, 32, 64 and 128; weight rows that are not whole tiles of 128; an odd number of blocks per row; one
# tile on a cluster of CTAs (long K); more tiles than SMs, shared between CTAs or dealt in turn.
@pytest.mark.parametrize("ggml_type,N,K,B", [
    (2, 128, 64, 16), (2, 100, 96, 17), (2, 256, 6912, 33), (2, 1152, 1056, 65), (2, 19200, 256, 9), (2, 6000, 320, 129), (2, 1536, 1152, 200),
    (2, 200, 128, 1025), (8, 256, 6912, 40), (8, 300, 96, 70), (8, 130, 1152, 300), (12, 256, 256, 16), (12, 129, 2304, 65), (12, 21504, 512, 32), (12, 384, 5376, 257)])
def test_gemm_tiles(gpu, ggml_type, N, K, B):
    """Relative error of a row below 5e-6: activations keep 22 bits (2^-22), and up to 33 additions of the tensor core are
    rounded towards zero, each by less than 2^-23 of the running sum, before the sum moves to registers."""
    rng = np.random.default_rng(N + K + B)
    raw = {2: gb.random_q4_0_blocks, 8: gb.random_q8_0_blocks, 12: gb.random_q4_k_blocks}[ggml_type](rng, N, K)
    x = rng.standard_normal((B, K), dtype=np.float32) * rng.uniform(0.01, 100.0, (B, 1)).astype(np.float32)
    before = gpu.tc_gemm_count()
    gpu.tc_gemm_policy(2)
    try:
        y = (_matmul(gpu, 8, A.DTYPE_GGUF_Q8_0, raw, N, K, x) if ggml_type == 8 else _gemv(gpu, ggml_type, raw, N, K, x)).astype(np.float64)
    finally:
        gpu.tc_gemm_policy(1)
    assert gpu.tc_gemm_count() == before + 1             # it is the GEMM that ran
    ref = x.astype(np.float64) @ q4_blocks.dequant(raw.reshape(-1), ggml_type, N, K).astype(np.float64).T
    assert (np.linalg.norm(y - ref, axis=1) / np.linalg.norm(ref, axis=1)).max() < 5e-6
    assert gpu.device_error() == 0


# Tiles of 256 rows, where the estimate of launch_rows prefers them: whole tiles with a ragged last one in both directions, a K of an
# odd number of steps; tiles shared between CTAs (the last two).
@pytest.mark.parametrize("ggml_type,N,K,B,shared", [
    (2, 18944, 256, 512, 0), (2, 18900, 2112, 449, 0), (2, 18944, 96, 385, 0), (12, 18944, 1792, 512, 0), (12, 21504, 5376, 1024, 1),
    (2, 21487, 2560, 1000, 1)])
def test_gemm_tiles_of_256_rows(gpu, ggml_type, N, K, B, shared):
    """Two steps' main terms between read-outs, the cross terms added first: eight additions at full magnitude, each rounded
    towards zero by less than 2^-23 of the sum so far: at most 2^-23 * (1 + .. + 8) / 8 = 5.4e-7 of the two steps' sum, half of it
    on average; no further from the exact product than the three steps of the smaller tiles (2.8e-7 measured)."""
    rng = np.random.default_rng(N + K + B)
    raw = {2: gb.random_q4_0_blocks, 12: gb.random_q4_k_blocks}[ggml_type](rng, N, K)
    x = rng.standard_normal((B, K), dtype=np.float32) * rng.uniform(0.01, 100.0, (B, 1)).astype(np.float32)
    before = gpu.gemm_counts()
    y = _gemv(gpu, ggml_type, raw, N, K, x).astype(np.float64)
    after = gpu.gemm_counts()
    assert after["tile_256"] == before["tile_256"] + 1 and after["shared"] == before["shared"] + shared
    ref = x.astype(np.float64) @ q4_blocks.dequant(raw.reshape(-1), ggml_type, N, K).astype(np.float64).T
    print(f"error {np.linalg.norm(y - ref) / np.linalg.norm(ref):.2e}, worst row {(np.linalg.norm(y - ref, axis=1) / np.linalg.norm(ref, axis=1)).max():.2e}")
    assert (np.linalg.norm(y - ref, axis=1) / np.linalg.norm(ref, axis=1)).max() < 1e-6
    assert np.linalg.norm(y - ref) < 5.4e-7 * np.linalg.norm(ref)
    assert np.linalg.norm(y - ref) < 3e-7 * np.linalg.norm(ref) or ggml_type == 12
    assert gpu.device_error() == 0


# Products that 128-row tiles as clusters would take several waves for.
@pytest.mark.parametrize("N,K,B", [(1152, 1024, 1280), (1536, 1152, 1800), (1152, 6912, 1280), (4096, 2560, 300), (2560, 2048, 1024)])
def test_clusters_run_in_one_wave(gpu, N, K, B):
    """Clusters of CTAs that share a K are for calls whose tiles leave SMs idle: never more of them than run at once.  Error as in
    test_gemm_tiles."""
    rng = np.random.default_rng(N + K + B)
    raw = gb.random_q4_0_blocks(rng, N, K)
    x = rng.standard_normal((B, K), dtype=np.float32)
    before = gpu.gemm_counts()
    y = _gemv(gpu, 2, raw, N, K, x).astype(np.float64)
    after = gpu.gemm_counts()
    assert after["tile_128"] + after["tile_256"] > before["tile_128"] + before["tile_256"] and after["cluster_waves"] == before["cluster_waves"]
    ref = x.astype(np.float64) @ q4_blocks.dequant(raw.reshape(-1), 2, N, K).astype(np.float64).T
    assert (np.linalg.norm(y - ref, axis=1) / np.linalg.norm(ref, axis=1)).max() < 5e-6 and gpu.device_error() == 0


def _gemm_error(gpu, ggml_type, raw, N, K, x):
    """Errors against float64, as 2-norms over the result's: of the GEMM, and of the GEMV that takes its place where it is refused."""
    ref = x.astype(np.float64) @ q4_blocks.dequant(raw.reshape(-1), ggml_type, N, K).astype(np.float64).T
    errors = []
    for policy in (2, 0):
        before = gpu.tc_gemm_count()
        gpu.tc_gemm_policy(policy)
        try:
            y = _gemv(gpu, ggml_type, raw, N, K, x, tile=N % 16 == 0 and K % 64 == 0).astype(np.float64)
        finally:
            gpu.tc_gemm_policy(1)
        assert (gpu.tc_gemm_count() > before) == (policy == 2)
        errors.append(np.linalg.norm(y - ref) / np.linalg.norm(ref))
    return errors


@pytest.mark.parametrize("N,K,B", [(256, 5376, 9), (129, 2304, 40), (256, 21504, 64), (384, 5376, 130)])
def test_gemm_q4_k_activations_with_a_mean(gpu, N, K, B):
    """Q4_K codes are not negative and a block's minimum is taken off afterwards: with activations that have a mean, the two
    parts are some 60 times the result here.  Same bound as for the tiles: the sums must not be larger than the result."""
    rng = np.random.default_rng(K + B)
    raw = rng.integers(0, 256, (N * K // 256, 144), dtype=np.uint8)
    d = ((0.5 + rng.random((len(raw), 1))) * 1e-4).astype(np.float16)
    raw[:, 0:2], raw[:, 2:4] = d.view(np.uint8), (d * np.float16(7.5)).view(np.uint8)
    assert _gemm_error(gpu, 12, raw, N, K, rng.standard_normal((B, K), dtype=np.float32) + np.float32(1))[0] < 5e-6


@pytest.mark.parametrize("ggml_type,N,K,B", [(2, 512, 1152, 9), (2, 512, 1152, 33), (2, 256, 6912, 64), (2, 512, 1152, 65), (12, 256, 5376, 16), (12, 256, 5376, 40),
                                             (12, 256, 21504, 129)])
def test_gemm_is_as_close_as_the_gemv(gpu, ggml_type, N, K, B):
    """The tensor core rounds its sums towards zero, so the GEMM moves them to registers every few additions; it has to end no
    further from the exact product than the GEMV (exact integer sums per block) whose calls it takes."""
    rng = np.random.default_rng(N + K + B)
    raw = {2: gb.random_q4_0_blocks, 12: gb.random_q4_k_blocks}[ggml_type](rng, N, K)
    gemm, gemv = _gemm_error(gpu, ggml_type, raw, N, K, rng.standard_normal((B, K), dtype=np.float32))
    assert gemm <= gemv


@pytest.mark.parametrize("B", [3, 4, 9, 64, 130])
def test_q8_0_products_are_fp32_sums(gpu, B):
    """A Q8_0 product of many rows: 1152 / 32 additions per lane and five between lanes, each rounded to nearest, end about
    2^-24 * sqrt(41 / 3) * 2/3 = 1.5e-7 from the exact product."""
    rng = np.random.default_rng(B)
    N, K = 1024, 1152
    raw, x = gb.random_q8_0_blocks(rng, N, K), rng.standard_normal((B, K), dtype=np.float32)
    y = _matmul(gpu, 8, A.DTYPE_GGUF_Q8_0, raw, N, K, x).astype(np.float64)
    ref = x.astype(np.float64) @ q4_blocks.dequant(raw.reshape(-1), 8, N, K).astype(np.float64).T
    assert np.linalg.norm(y - ref) < 1.5e-7 * np.linalg.norm(ref)


@pytest.mark.parametrize("ggml_type,K,scale", [(2, 256, 9000.0), (2, 256, -65504.0), (12, 512, 200.0), (12, 512, 65504.0)])
def test_weights_beyond_fp16(gpu, ggml_type, K, scale):
    """One block whose weights fp16 cannot hold, among ordinary ones: many rows of activations give what the GEMV gives for one."""
    N, B = 64, 16
    rng = np.random.default_rng(K)
    raw = {2: gb.random_q4_0_blocks, 12: gb.random_q4_k_blocks}[ggml_type](rng, N, K).copy()
    blocks = raw.reshape(-1, {2: 18, 12: 144}[ggml_type])
    blocks[7, 0:2] = np.array([scale], np.float16).view(np.uint8)
    x = rng.standard_normal((B, K), dtype=np.float32)
    y = _gemv(gpu, ggml_type, raw, N, K, x).astype(np.float64)
    ref = x.astype(np.float64) @ q4_blocks.dequant(raw.reshape(-1), ggml_type, N, K).astype(np.float64).T
    assert (np.linalg.norm(y - ref, axis=0) <= 2e-5 * np.linalg.norm(ref, axis=0)).all()
    # over the row-tiled copy: the few-row kernel, which has no such limit
    before = gpu.gemm_counts()
    y = _gemv(gpu, ggml_type, raw, N, K, x[:7], tile=True).astype(np.float64)
    after = gpu.gemm_counts()
    assert after["few"] == before["few"] + 1 and after["tile_16"] == before["tile_16"]
    assert (np.linalg.norm(y - ref[:7], axis=0) <= 2e-5 * np.linalg.norm(ref[:7], axis=0)).all()


def test_gemm_calls_from_several_threads(gpu):
    """Products of four threads share one image of activations; each thread has a map, handles and rows of its own."""
    import threading
    rng, N, K, B, wrong = np.random.default_rng(9), 256, 512, 16, []
    raw = gb.random_q4_0_blocks(rng, N, K)
    W = q4_blocks.dequant(raw.reshape(-1), 2, N, K).astype(np.float64)
    gpu.map_create_typed(91, A.DTYPE_GGUF_Q4_0, 1, N * K)
    gpu.upload_gguf_blocks(91, 2, 0, raw)
    locs = [gpu.upload_dev(np.array([v], np.uint32))[0] for v in (0, 0, B * K)]

    def work(k):
        rng = np.random.default_rng(k)
        for i in range(100):
            x = rng.standard_normal((B, K), dtype=np.float32)
            gpu.scatter_contiguous(80 + k, 0, x)
            gpu.map_matmul_t_xq4_dev(80 + k, 91, locs[0], locs[1], locs[2], B, K, N)
            y = gpu.gather(80 + k, np.arange(B * K, B * K + B * N, dtype=np.uint32)).view(np.float32).reshape(B, N)
            ref = x.astype(np.float64) @ W.T
            if np.linalg.norm(y - ref) > 5e-6 * np.linalg.norm(ref):
                wrong.append((k, i))

    before = gpu.tc_gemm_count()
    for k in range(4):
        gpu.map_create_typed(80 + k, A.DTYPE_F32, 1, B * K + B * N)
    try:
        threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not wrong and gpu.device_error() == 0 and gpu.tc_gemm_count() == before + 400
    finally:
        for k in range(4):
            gpu.map_destroy(80 + k)
        gpu.map_destroy(91)
        for h in locs:
            gpu.free_handle(h)


@pytest.mark.parametrize("batch", [9, 17, 40])
def test_batched_head_and_ragged_prefill_match_the_oracle(gpu, batch):
    """Prompts of 1 to 70 tokens through one ragged prefill, then steps whose products and arg-max are the GEMM's."""
    cfg = tiny_gemma3(n_layer=2, n_vocab=1000)
    tensors = synth.build_model(cfg, gb.GGML_TYPE_Q4_0, seed=61, tied=False)
    f32 = dequant_model(tensors)
    lens = [1 + (23 * i) % 70 for i in range(batch)]
    prompts = [synth.random_prompt(cfg.n_vocab, n, seed=100 + i) for i, n in enumerate(lens)]
    eng = ADAMEngine(gpu, cfg, tensors, kv_cap=80, kv_dtype="f32", max_batch=batch)
    try:
        eng.begin(prompts, [max(lens) + 3] * batch)
        eng.step(1, lm_head=False)
        before = gpu.tc_gemm_count()
        eng.step(1, lm_head=True, direct=True)
        assert gpu.tc_gemm_count() == before + 4 * cfg.n_layer + 1          # four products per layer and the head
        outs, _ = eng.generate_batch(prompts, GenerationConfig(max_tokens=3, **GREEDY))
        for p, o in list(zip(prompts, outs))[:: max(1, batch // 8)]:
            assert o == OracleDecoder(cfg, f32, kv_cap=80).generate(p, 3)[0]
        assert gpu.device_error() == 0
    finally:
        eng.close()


def test_host_sampling_of_a_ragged_batch_draws_in_step_order(gpu):
    """Sequences that are sampled on the host share one seeded random stream: one whose prompt is longer by n tokens draws its
    first number n steps later, and within a step they draw in their order."""
    cfg = tiny_gemma3(n_layer=1, n_vocab=64)
    tensors = synth.build_model(cfg, gb.GGML_TYPE_Q4_0, seed=66)
    prompts = [list(synth.random_prompt(cfg.n_vocab, n, seed=n)) for n in (7, 3, 5)]
    rule = GenerationConfig(max_tokens=5, eos_token_ids=(), temperature=1.0, top_k=0, top_p=1.0, repeat_penalty=1.0, seed=11)
    eng = ADAMEngine(gpu, cfg, tensors, kv_cap=32, kv_dtype="f32", max_batch=3)
    try:
        outs, stats = eng.generate_batch(prompts, rule)
        assert stats["sampling_mode"] == "cpu"
        rng, want = np.random.default_rng(11), [[] for _ in prompts]
        for step in range(4 + 5):
            for b, p in enumerate(prompts):
                if len(p) - 3 <= step and len(want[b]) < 5:
                    want[b].append(eng._sample(eng.logits_trace(p + want[b])[-1], rule, [], rng))
        assert outs == want
    finally:
        eng.close()


# Query rows per attention tile: 32 (a chunk that does not fill the GPU), 64 and 128 (it does); windows and pages whose edges
# lie inside a cache tile; prompts longer than one chunk of 2048 rows (n_embd 128), cut inside a sequence.
@pytest.mark.parametrize("kv_dtype", ["f16", "f32"])
@pytest.mark.parametrize("head_dim,n_head,n_kv,window,lens", [
    (256, 4, 1, 0, (14, 66, 193)), (128, 2, 1, 40, (129, 3, 64)), (64, 8, 1, 0, (65, 33)), (32, 4, 4, 24, (100, 2)),
    (64, 16, 8, 0, (700, 500)), (32, 32, 16, 100, (1300,)), (64, 16, 8, 0, (1300, 1000)), (32, 32, 16, 100, (2300,))])
def test_prompt_attention_tiles(gpu, head_dim, n_head, n_kv, window, lens, kv_dtype):
    """The token after the prompts has the logits of single steps.  f32 cache: 2e-5 (both sides sum in fp32, in different
    orders); f16: a last-bit difference can move a cached value by one f16 step."""
    cfg = tiny_gemma3(n_layer=2, n_embd=128, n_head=n_head, n_head_kv=n_kv, head_dim=head_dim, n_ff=128, n_vocab=256, sliding_window=window)
    tensors = synth.build_model(cfg, gb.GGML_TYPE_Q4_0, seed=62)
    prompts = [synth.random_prompt(cfg.n_vocab, n, seed=70 + n) for n in lens]
    eng = ADAMEngine(gpu, cfg, tensors, kv_cap=max(lens) + 8, kv_dtype=kv_dtype, max_batch=len(lens), window=window > 0)
    try:
        eng.begin(prompts, [max(lens) + 2] * len(lens))  # first: the steps would leave the right keys and values in the cache
        gpu.batch_begin(); eng.prefill_prompts(prompts, 0); eng.step(1, lm_head=True, logits=True); gpu.batch_end()
        got = [eng.read_logits(b) for b in range(len(lens))]
        want = []
        for p in prompts:
            eng.begin([p], [len(p) + 2])
            gpu.batch_begin(); eng.step(len(p) - 1, lm_head=False); eng.step(1, lm_head=True, logits=True); gpu.batch_end()
            want.append(eng.read_logits(0))
        tol = 1e-3 if kv_dtype == "f16" else 2e-5
        for g, w in zip(got, want):
            assert np.abs(g - w).max() <= tol * np.abs(w).max()
        assert gpu.device_error() == 0
    finally:
        eng.close()


@pytest.mark.parametrize("n", [1, 2, 65, 130])
def test_score_equals_steps(gpu, n):
    cfg = replace(tiny_gemma3(n_layer=2), n_vocab=512)
    tensors = synth.build_model(cfg, gb.GGML_TYPE_Q4_0, seed=63)
    toks = synth.random_prompt(cfg.n_vocab, n, seed=5)
    eng = ADAMEngine(gpu, cfg, tensors, kv_cap=160, kv_dtype="f32")
    try:
        got = eng.logits_trace(toks)                     # first: the steps would leave the right keys and values in the cache
        eng.begin([toks], [n])
        want = []
        for _ in range(n):
            eng.step(1, lm_head=True, logits=True)
            want.append(eng.read_logits(0))
        want = np.stack(want)
        assert np.abs(got - want).max() <= 2e-5 * np.abs(want).max()
    finally:
        eng.close()


@pytest.mark.parametrize("n,embd_type", [(1, None), (64, None), (65, 8), (130, None)])
def test_score_leaves_the_decoder_as_steps_do(gpu, n, embd_type):
    """Logits, token, position, log and last rows after scoring, and the step that follows, are those of n single steps."""
    cfg = replace(tiny_gemma3(n_layer=2), n_vocab=512)
    tensors = synth.build_model(cfg, gb.GGML_TYPE_Q4_0, seed=64, embd_type=embd_type)
    toks = synth.random_prompt(cfg.n_vocab, n, seed=6)
    eng = ADAMEngine(gpu, cfg, tensors, kv_cap=160, kv_dtype="f32")

    def state():
        pos, tok = eng.read_state()
        return int(pos[0]), int(tok[0]), eng.read_log(0, 1, n).tolist(), eng.read_logits(0), eng.read_buffer(0, cfg.n_embd)

    try:
        seen = []
        for scored in (False, True):
            eng.begin([synth.random_prompt(cfg.n_vocab, 3, seed=7)], [4])       # other logits in the buffers beforehand
            eng.step(3, lm_head=True, logits=True)
            eng.begin([toks], [n + 2])
            if scored:
                eng._score(n, True)
            else:
                eng.step(n, lm_head=True, logits=True)
            after = state()
            eng.step(1, lm_head=True, logits=True)
            seen.append((after, state()))
        for (p0, t0, l0, y0, h0), (p1, t1, l1, y1, h1) in zip(*seen):
            assert (p0, t0, l0) == (p1, t1, l1)
            assert np.abs(y0 - y1).max() <= 2e-5 * np.abs(y0).max() and np.abs(h0 - h1).max() <= 2e-5 * np.abs(h0).max()
        assert gpu.device_error() == 0
    finally:
        eng.close()


@pytest.mark.parametrize("max_batch,left_mb", [(1, 8), (3, 8), (1, 100)])
def test_score_without_room_for_its_buffer(gpu, max_batch, left_mb):
    """Two groups of 64 rows of 131072 logits are 67 MB: with less on the device the groups get smaller, down to the logits
    buffer of the decoder, which single steps never needed more than."""
    import torch
    cfg = replace(tiny_gemma3(n_layer=1), n_vocab=131072)
    tensors = synth.build_model(cfg, gb.GGML_TYPE_Q4_0, seed=65)
    toks = synth.random_prompt(cfg.n_vocab, 70, seed=8)
    want, filler = None, None
    for full in (False, True):
        eng = ADAMEngine(gpu, cfg, tensors, kv_cap=80, kv_dtype="f32", max_batch=max_batch)
        try:
            if full:
                eng.begin([toks], [70])
                eng.prefill(3)                           # the buffers of a prompt exist
                torch.cuda.empty_cache()
                filler = torch.empty(torch.cuda.mem_get_info()[0] - (left_mb << 20), dtype=torch.uint8, device="cuda")
            got = eng.logits_trace(toks)
            assert np.array_equal(eng.read_logits(0), got[-1])
            assert gpu.device_error() == 0
        finally:
            del filler
            filler = None
            torch.cuda.empty_cache()
            eng.close()
        if want is None:
            want = got
    assert np.abs(got - want).max() <= 2e-5 * np.abs(want).max()


def test_decoder_where_a_full_chunk_of_rows_does_not_fit(gpu):
    """1024 rows of this model's activations take 67 MB; with 56 MB left on the device, enough for the model and the 64 rows that a
    decoder cannot do without, it has smaller chunks and the same results."""
    import torch
    cfg = replace(tiny_gemma3(n_layer=1), n_ff=16384)
    tensors = synth.build_model(cfg, gb.GGML_TYPE_Q4_0, seed=67)
    toks = synth.random_prompt(cfg.n_vocab, 600, seed=9)
    seen, filler, eng = [], None, None
    for full in (False, True):
        try:
            if full:
                torch.cuda.empty_cache()
                filler = torch.empty(torch.cuda.mem_get_info()[0] - (56 << 20), dtype=torch.uint8, device="cuda")
            eng = ADAMEngine(gpu, cfg, tensors, kv_cap=1024, kv_dtype="f32")
            eng.begin([toks], [602])
            eng.prefill(599)
            eng.step(1, lm_head=True, logits=True)
            seen.append(eng.read_logits(0))
            assert gpu.device_error() == 0
        finally:
            del filler
            filler = None
            torch.cuda.empty_cache()
            if eng is not None:
                eng.close()
                eng = None
    assert np.abs(seen[0] - seen[1]).max() <= 2e-5 * np.abs(seen[0]).max()


@pytest.mark.parametrize("n", [1, 16383, 16384, 262144, 262145, 1200000])
def test_large_results_and_uploads(gpu, n):
    """Around the sizes where results move to page-locked blocks and uploads leave the ring; neighbouring locs and others; arrays
    that outlive the next call keep their values."""
    gpu.map_create_typed(90, A.DTYPE_F32, 1, 1300000)
    try:
        x = np.random.default_rng(n).standard_normal(n + 7).astype(np.float32)
        gpu.scatter_contiguous(90, 0, x)
        locs = np.arange(n, dtype=np.uint32)
        first = gpu.gather(90, locs + 7).view(np.float32)
        swapped = locs.copy()
        swapped[n // 2:] = swapped[n // 2:][::-1]
        mixed = gpu.gather(90, swapped).view(np.float32)
        near = locs.copy()
        if n > 2:
            near[n // 2] = 0                            # first and last as if they were neighbours
        almost = gpu.gather(90, near).view(np.float32)
        assert np.array_equal(first, x[7:]) and np.array_equal(mixed, x[swapped]) and np.array_equal(almost, x[near])
        del first, mixed, almost
        gc.collect()
        kept = [gpu.gather(90, locs).view(np.float32) for _ in range(3)]
        gpu.scatter_contiguous(90, 0, -x)
        again = gpu.gather(90, locs).view(np.float32)
        assert all(np.array_equal(k, x[:n]) for k in kept) and np.array_equal(again, -x[:n])
    finally:
        gpu.map_destroy(90)


@pytest.mark.parametrize("n", [5, 20000, 1100000])
def test_gather_onto_its_own_locs(gpu, n):
    """The result may overwrite the locs: neighbours, and locs that only look like neighbours at both ends; results that go
    through the staging buffer, and larger ones."""
    gpu.map_create_typed(90, A.DTYPE_F32, 1, n)
    try:
        x = np.random.default_rng(n).standard_normal(n).astype(np.float32)
        gpu.scatter_contiguous(90, 0, x)
        swapped = np.arange(n, dtype=np.uint32)
        swapped[1:-1] = swapped[1:-1][::-1]
        for locs in (np.arange(n, dtype=np.uint32), swapped):
            want = x[locs]
            assert gpu._lib.map_gather(90, locs.ctypes.data, locs.ctypes.data, n) == 0
            assert np.array_equal(locs.view(np.float32), want)
        assert gpu.device_error() == 0
    finally:
        gpu.map_destroy(90)


def test_host_io_from_several_threads(gpu):
    """Each thread writes and reads a map of its own, over all sizes of the staging; the copies run outside Python's lock."""
    import threading
    wrong = []

    def work(k):
        rng = np.random.default_rng(k)
        for i in range(60):
            n = int(rng.choice([3, 1000, 20000, 300000]))
            x, locs = rng.standard_normal(n).astype(np.float32), rng.permutation(n).astype(np.uint32)
            gpu.scatter(80 + k, locs, x)
            whole, mixed = gpu.gather(80 + k, np.arange(n, dtype=np.uint32)).view(np.float32), gpu.gather(80 + k, locs).view(np.float32)
            if not (np.array_equal(whole[locs], x) and np.array_equal(mixed, x)):
                wrong.append((k, i, n))

    for k in range(4):
        gpu.map_create_typed(80 + k, A.DTYPE_F32, 1, 300000)
    try:
        threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not wrong and gpu.device_error() == 0
    finally:
        for k in range(4):
            gpu.map_destroy(80 + k)


@pytest.mark.parametrize("N", [8192, 8193, 70001, 300000])
def test_argmax_of_one_row_on_several_ctas(gpu, N):
    """A Q8_0 head's winner, and of equal rows that different CTAs look at the first."""
    K, first, second = 64, N // 3, N - 1
    rng = np.random.default_rng(N)
    raw = gb.random_q8_0_blocks(rng, N, K).reshape(N, -1).copy()
    x = rng.standard_normal(K).astype(np.float32)
    y = q4_blocks.dequant(raw.reshape(-1), 8, N, K).astype(np.float64) @ x
    raw[first] = raw[second] = raw[int(y.argmax())].copy()
    want = min(first, int(y.argmax()))
    gpu.map_create_typed(91, A.DTYPE_GGUF_Q8_0, 1, N * K)
    gpu.upload_gguf_blocks(91, 8, 0, raw.reshape(-1))
    gpu.map_create_typed(90, A.DTYPE_F32, 1, K + 4)
    locs = [gpu.upload_dev(np.array([v], np.uint32))[0] for v in (0, 0, K)]
    try:
        gpu.scatter_contiguous(90, 0, x)
        for _ in range(2):
            with gpu.batch():
                gpu.map_matvec_argmax_t_xq4_dev(90, 91, locs[0], locs[1], locs[2], locs[2], locs[2], K, N)
            assert int(gpu.gather(90, np.array([K], np.uint32)).view(np.float32)[0]) == want
    finally:
        for h in locs:
            gpu.free_handle(h)
        gpu.map_destroy(90)
        gpu.map_destroy(91)
