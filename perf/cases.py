"""Timed cases of the quantized decode path, through the package's public entry points.

Three kinds of program use the package, and each kind has its cases:

* ``generate``: a chat or batch server.  ``ADAMEngine.generate`` / ``generate_batch`` over a loaded model: prompt
  ids in from the host, prefill, decode, sampled ids back on the host.
* ``score``: evaluation.  ``ADAMEngine.logits_trace``: the logits after every position of a given text.
* ``ffn`` and ``lm_head``: a host engine that issues the backend's operators one by one, as the reference engine
  does: activations uploaded, a feed-forward block (norm, gate, up, GeGLU, down, norm + residual) or an LM head with
  arg-max in one batch, the result read back.

Models have the Gemma-3-1B shape (26 layers, Q4_0 or Q4_0 with a Q8_0 embedding table, which is how real files store
it) and the Gemma-3-27B shape cut to 8 of its 62 layers (Q4_K), with random weights.  A model is loaded once per
process and kept, as a server keeps it; a case's inputs (token ids, activations) come from the seed.
"""
import math
import weakref

import numpy as np
import torch

import adam_b200 as A
from adam_b200 import synth
from adam_b200.config import GenerationConfig, gemma3_1b, gemma3_27b, with_layers
from adam_b200.engine import ADAMEngine

Q4_0, Q4_K, Q8_0 = A.GGML_TYPE_Q4_0, A.GGML_TYPE_Q4_K, 8
TYPES = {"q4_0": Q4_0, "q4_k": Q4_K, "q8_0": Q8_0}
MAP_DTYPE = {"q4_0": A.DTYPE_GGUF_Q4_0, "q4_k": A.DTYPE_GGUF_Q4_K, "q8_0": 18}
BLOCK = {"q4_0": (32, 18), "q4_k": (256, 144), "q8_0": (32, 34)}          # weights and bytes of a GGUF block

# ---- the cases ---------------------------------------------------------------------------------------------------


def listed():
    return [
        # one token through one feed-forward block, operator by operator: the smallest call sequence
        {"name": "ffn_q4_0_1row", "kind": "ffn", "type": "q4_0", "n_embd": 1152, "n_ff": 6912, "rows": 1},
        # a decode batch of eight at the 27B widths
        {"name": "ffn_q4_k_8rows", "kind": "ffn", "type": "q4_k", "n_embd": 5376, "n_ff": 21504, "rows": 8},
        # a prompt's rows through the block at once, an odd number of them
        {"name": "ffn_q4_0_201rows", "kind": "ffn", "type": "q4_0", "n_embd": 1152, "n_ff": 6912, "rows": 201},
        # next-token choice over the full vocabulary
        {"name": "lm_head_q4_0", "kind": "lm_head", "type": "q4_0", "n_vocab": 262144, "n_embd": 1152},
        # a short chat turn: a dozen ids in, a few out (time to the first tokens)
        {"name": "chat_1b_short", "kind": "generate", "model": "1b", "batch": 1, "shortest": 13, "longest": 13, "new": 6, "sampled": False},
        # the ordinary single-user request
        {"name": "chat_1b", "kind": "generate", "model": "1b", "batch": 1, "shortest": 128, "longest": 128, "new": 64, "sampled": False},
        # a long document and a short answer, default sampling rule (top-k, nucleus, repeat penalty)
        {"name": "document_1b_sampled", "kind": "generate", "model": "1b_q8", "batch": 1, "shortest": 1500, "longest": 1500, "new": 12, "sampled": True},
        # a full batch of 512-token prompts
        {"name": "batch32_1b", "kind": "generate", "model": "1b", "batch": 32, "shortest": 512, "longest": 512, "new": 24, "sampled": False},
        # a few users with prompts of different lengths
        {"name": "ragged7_1b", "kind": "generate", "model": "1b_q8", "batch": 7, "shortest": 21, "longest": 259, "new": 24, "sampled": False},
        # evaluation of a text
        {"name": "score_1b", "kind": "score", "model": "1b_q8", "tokens": 65},
        # the large model: one user, and a batch of 64
        {"name": "chat_27b", "kind": "generate", "model": "27b", "batch": 1, "shortest": 100, "longest": 100, "new": 24, "sampled": False},
        {"name": "batch64_27b", "kind": "generate", "model": "27b", "batch": 64, "shortest": 128, "longest": 128, "new": 12, "sampled": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ffn", "lm_head", "generate", "generate", "generate", "score"])
    if kind == "ffn":
        return {"kind": "ffn", "type": rng.choice(["q4_0", "q4_k"]), "n_embd": 256 * rng.randint(2, 21), "n_ff": 256 * _log(rng, 4, 84),
                "rows": _log(rng, 1, 512)}
    if kind == "lm_head":
        return {"kind": "lm_head", "type": rng.choice(["q4_0", "q4_k", "q8_0"]), "n_vocab": _log(rng, 8000, 262144), "n_embd": 256 * rng.randint(2, 21)}
    model = rng.choice(["1b", "1b_q8", "27b"])
    if kind == "score":
        return {"kind": "score", "model": model, "tokens": _log(rng, 16, 128)}
    sampled = rng.random() < 0.25
    batch = 1 if sampled else _log(rng, 1, 64)
    longest = _log(rng, 8, min(MODELS[model]["kv_cap"] - 64, 8192 // batch))
    shortest = longest if batch == 1 or rng.random() < 0.5 else rng.randint(max(1, longest // 4), longest)
    return {"kind": "generate", "model": model, "batch": batch, "shortest": shortest, "longest": longest,
            "new": _log(rng, 1, 12 if sampled else 24), "sampled": sampled}


# ---- models and operands that a program keeps ----------------------------------------------------------------------

MODELS = {
    "1b": dict(cfg=gemma3_1b(), type="q4_0", table="q4_0", kv_cap=2048, kv_dtype="f16"),
    "1b_q8": dict(cfg=gemma3_1b(), type="q4_0", table="q8_0", kv_cap=2048, kv_dtype="f32"),
    "27b": dict(cfg=with_layers(gemma3_27b(), 8), type="q4_k", table="q4_k", kv_cap=1024, kv_dtype="f16"),
}
MAX_BATCH = 64
_kept = {}
_free_maps = list(range(255, -1, -1))


def _gpu():
    if "gpu" not in _kept:
        _kept["gpu"] = A.init()
    return _kept["gpu"]


def _blocks(kind, rows, cols, gen):
    """Random GGUF blocks on the GPU.  Q4_0 and Q8_0: N(0, 0.02) weights, quantized; Q4_K, for which there is no encoder on
    the GPU: random codes and sub-scales, means near zero and the same spread."""
    per, nbytes = BLOCK[kind]
    n = rows * cols // per
    if kind == "q4_k":
        raw = torch.randint(0, 256, (n, nbytes), dtype=torch.uint8, device="cuda", generator=gen)
        d = ((0.5 + torch.rand((n, 1), device="cuda", generator=gen)) * (0.02 / 260.0)).to(torch.float16)
        raw[:, 0:2] = d.view(torch.uint8)
        raw[:, 2:4] = (d * 7.5).view(torch.uint8)               # value = d * scale * code - dmin * min, codes 7.5 on average
    else:
        raw = torch.empty((n, nbytes), dtype=torch.uint8, device="cuda")
        for i in range(0, n, 1 << 22):                          # bounded temporaries
            w = torch.randn((min(n - i, 1 << 22), per), device="cuda", generator=gen) * 0.02
            if kind == "q4_0":
                torch.cuda.synchronize()
                _gpu().quantize_q4_0_dev(w.data_ptr(), w.numel(), raw[i:].data_ptr())
            else:
                d = w.abs().amax(1, keepdim=True) / 127.0
                raw[i:i + len(w), 0:2] = d.to(torch.float16).view(torch.uint8)
                raw[i:i + len(w), 2:] = (w / d).round().to(torch.int8).view(torch.uint8)
    torch.cuda.synchronize()
    return synth.QTensor(TYPES[kind], rows, cols, raw.reshape(-1))


def _engine(name):
    if name in _kept:
        return _kept[name]
    gpu, m = _gpu(), MODELS[name]
    cfg, gen = m["cfg"], torch.Generator(device="cuda").manual_seed(len(name))

    def norm(n):
        return (1.0 + 0.1 * torch.randn(n, device="cuda", generator=gen)).cpu().numpy()

    t = {"token_embd.weight": _blocks(m["table"], cfg.n_vocab, cfg.n_embd, gen), "output_norm.weight": norm(cfg.n_embd)}
    for layer in range(cfg.n_layer):
        for n in synth.LAYER_NORMS:
            t[f"blk.{layer}.{n}.weight"] = norm(cfg.n_embd)
        for n in ("attn_q_norm", "attn_k_norm"):
            t[f"blk.{layer}.{n}.weight"] = norm(cfg.head_dim)
        for n, (rows, cols) in synth.mat_shapes(cfg).items():
            t[f"blk.{layer}.{n}.weight"] = _blocks(m["type"], rows, cols, gen)
    n_maps = cfg.n_layer + 2                                     # one per layer, the embedding table, the norms
    ids = sorted(_free_maps[-n_maps:])
    del _free_maps[-n_maps:]
    engine = type("Engine", (ADAMEngine,), {"WS_MAP": ids[0], "FIRST_WT_MAP": ids[1]})
    _kept[name] = engine(gpu, cfg, t, kv_cap=m["kv_cap"], max_batch=MAX_BATCH, kv_dtype=m["kv_dtype"], window=True)
    _kept[name].tensors = {}
    return _kept[name]


class _Held:
    """Maps and loc handles of one program, given back with it."""

    def __init__(self):
        self.gpu, self.maps, self.handles = _gpu(), [], []
        self._end = weakref.finalize(self, _Held._release, self.gpu, self.maps, self.handles)

    def map(self, dtype, n):
        self.maps.append(_free_maps.pop())
        self.gpu.map_create_typed(self.maps[-1], dtype, 1, n)
        return self.maps[-1]

    def loc(self, values):
        h, _ = self.gpu.upload_dev(np.ascontiguousarray(values, np.uint32))
        self.handles.append(h)
        return h

    def weights(self, kind, mats, gen):
        """One map with the matrices back to back, their row-tiled copies where the shape has one; their element offsets."""
        m, offs = self.map(MAP_DTYPE[kind], sum(r * c for r, c in mats)), []
        for rows, cols in mats:
            offs.append(offs[-1] + prev if offs else 0)
            prev = rows * cols
            q = _blocks(kind, rows, cols, gen)
            self.gpu.upload_gguf_blocks(m, q.ggml_type, offs[-1], int(q.raw.data_ptr()), int(q.raw.numel()))
            if kind != "q8_0" and rows % 16 == 0:
                self.gpu.tile_tensor(m, offs[-1], rows, cols)
        return m, offs

    @staticmethod
    def _release(gpu, maps, handles):
        for h in handles:
            gpu.free_handle(h)
        for m in maps:
            gpu.map_destroy(m)
            _free_maps.append(m)


# ---- prepare and run -------------------------------------------------------------------------------------------------


def _lengths(case):
    """Prompt lengths of a batch, evenly spread between the shortest and the longest, in a mixed order."""
    n = np.linspace(case["shortest"], case["longest"], case["batch"]).round().astype(int)
    return [int(n[(5 * i + 2) % len(n)]) for i in range(len(n))] if len(n) % 5 else [int(v) for v in n]


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] in ("generate", "score"):
        eng = _engine(case["model"])
        lens = _lengths(case) if case["kind"] == "generate" else [case["tokens"]]
        prompts = [rng.integers(0, eng.cfg.n_vocab, n).tolist() for n in lens]
        s = {"kind": case["kind"], "engine": eng, "prompts": prompts}
        if case["kind"] == "generate":
            rule = dict(temperature=0.8, top_k=40, top_p=0.95, repeat_penalty=1.1, seed=seed) if case["sampled"] else \
                dict(temperature=0.0, top_k=1, repeat_penalty=1.0)
            s["config"] = GenerationConfig(max_tokens=case["new"], eos_token_ids=(), **rule)
        return s
    held, gen = _Held(), torch.Generator(device="cuda").manual_seed(seed)
    E, s = case["n_embd"], {"kind": case["kind"], "held": held, "type": case["type"]}
    if case["kind"] == "lm_head":
        V = case["n_vocab"]
        s["w"], _ = held.weights(case["type"], [(V, E)], gen)
        # activations: hidden state, norm weights, normed state, winner
        s["act"] = held.map(A.DTYPE_F32, 3 * E + 4)
        s["norm"] = (1.0 + 0.1 * rng.standard_normal(E)).astype(np.float32)
        held.gpu.scatter_contiguous(s["act"], E, s["norm"])
        s["x"] = rng.standard_normal(E).astype(np.float32)
        s["locs"] = {k: held.loc([v]) for k, v in {"x": 0, "norm": E, "y": 2 * E, "w": 0, "out": 3 * E}.items()}
        s["read"] = np.array([3 * E], np.uint32)
        s["shape"] = (E, V)
        return s
    F, M = case["n_ff"], case["rows"]
    s["w"], offs = held.weights(case["type"], [(F, E), (F, E), (E, F)], gen)
    s["weights"] = [held.loc([o]) for o in offs]
    # activations: residual stream, two norms, normed stream, gate, up, down, result
    at, n = {}, 0
    for k, size in (("x", M * E), ("pre", E), ("post", E), ("y", M * E), ("gate", M * F), ("up", M * F), ("down", M * E), ("out", M * E)):
        at[k], n = n, n + size
    s["act"] = held.map(A.DTYPE_F32, n)
    held.gpu.scatter_contiguous(s["act"], at["pre"], (1.0 + 0.1 * rng.standard_normal(2 * E)).astype(np.float32))
    s["x"] = rng.standard_normal((M, E)).astype(np.float32)
    s["locs"] = {k: held.loc([at[k]]) for k in ("y", "gate", "up", "down")}
    s["rows"] = {k: held.loc(at[k] + E * np.arange(M)) for k in ("x", "y", "down", "out")}
    s["norms"] = {k: held.loc(np.full(M, at[k])) for k in ("pre", "post")}
    s["each"] = {k: held.loc(at[k] + np.arange(M * F)) for k in ("gate", "up")}
    s["read"] = np.arange(at["out"], at["out"] + M * E, dtype=np.uint32)
    s["shape"] = (M, E, F)
    return s


def run(s):
    if s["kind"] == "generate":
        outs, _ = s["engine"].generate_batch(s["prompts"], s["config"])
        return np.array(outs, np.int32)
    if s["kind"] == "score":
        return s["engine"].logits_trace(s["prompts"][0])
    g, act, w, loc = s["held"].gpu, s["act"], s["w"], s["locs"]
    g.scatter_contiguous(act, 0, s["x"])
    if s["kind"] == "lm_head":
        E, V = s["shape"]
        with g.batch():
            g.map_rmsnorm_dev(act, loc["x"], loc["norm"], loc["y"], 1, E, 1e-6)
            g.map_matvec_argmax_t_xq4_dev(act, w, loc["y"], loc["w"], loc["out"], loc["out"], loc["out"], E, V)
        return g.gather(act, s["read"]).view(np.float32).astype(np.int32)
    M, E, F = s["shape"]
    rows, norms, each, (gate, up, down) = s["rows"], s["norms"], s["each"], s["weights"]
    with g.batch():
        g.map_rmsnorm_dev(act, rows["x"], norms["pre"], rows["y"], M, E, 1e-6)
        g.map_matmul_t_xq4_dev(act, w, loc["y"], gate, loc["gate"], M, E, F)
        g.map_matmul_t_xq4_dev(act, w, loc["y"], up, loc["up"], M, E, F)
        g.map_op2_dev(act, A.OP_GEGLU, each["gate"], each["up"], each["gate"], M * F)
        g.map_matmul_t_xq4_dev(act, w, loc["gate"], down, loc["down"], M, F, E)
        g.map_rmsnorm_add_dev(act, rows["down"], norms["post"], rows["x"], rows["out"], M, E, 1e-6)
    return g.gather(act, s["read"]).view(np.float32).reshape(M, E)


# ---- what a pass cannot do without -----------------------------------------------------------------------------------


def _bytes(kind, n):
    per, nbytes = BLOCK[kind]
    return n // per * nbytes


def work(case):
    if case["kind"] == "lm_head":
        V, E = case["n_vocab"], case["n_embd"]
        return {"bytes": _bytes(case["type"], V * E) + 8 * E + 4, "flops": 2 * V * E}
    if case["kind"] == "ffn":
        M, E, F = case["rows"], case["n_embd"], case["n_ff"]
        return {"bytes": 3 * _bytes(case["type"], E * F) + 8 * M * E + 8 * E, "flops": 6 * M * E * F}
    m = MODELS[case["model"]]
    cfg = m["cfg"]
    layer = sum(r * c for r, c in synth.mat_shapes(cfg).values())
    head = cfg.n_vocab * cfg.n_embd
    kv_row = 2 * cfg.n_head_kv * cfg.head_dim * (2 if m["kv_dtype"] == "f16" else 4)
    window = [cfg.n_ctx if cfg.is_global(i) else cfg.sliding_window for i in range(cfg.n_layer)]
    w_layers, w_head = cfg.n_layer * _bytes(m["type"], layer), _bytes(m["table"], head)
    if case["kind"] == "score":
        # the text's positions share one read of the weights; every position has its logits
        n = case["tokens"]
        seen = sum(sum(min(w, p + 1) for p in range(n)) for w in window)
        return {"bytes": w_layers + w_head + n * kv_row * cfg.n_layer + 4 * n * cfg.n_vocab,
                "flops": 2 * n * (cfg.n_layer * layer + head) + 4 * seen * cfg.n_head * cfg.head_dim}
    # a prompt but for its last token shares one read of the layers; every new token reads layers, head and cache again
    nbytes, flops = w_layers + case["new"] * (w_layers + w_head), 0
    for n in _lengths(case):
        end = n + case["new"]
        seen = sum(sum(min(w, p + 1) for p in range(end - 1)) for w in window)
        flops += 2 * ((end - 1) * cfg.n_layer * layer + case["new"] * head) + 4 * seen * cfg.n_head * cfg.head_dim
        nbytes += (end - 1) * cfg.n_layer * kv_row + sum(kv_row * min(w, p) for w in window for p in range(n, end))
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["kind"] == "ffn":
        return {"rel": 1e-5}                      # 32-bit sums behind two norms
    if case["kind"] == "score":
        # 32-bit activations through all layers; where keys and values are kept in 16 bits, what rounds differently there
        return {"rel": 5e-5 if MODELS[case["model"]]["kv_dtype"] == "f32" else 1e-3}
    return {"rel": 0.0, "differ": 0.01}           # ids: two candidates may tie to the last bits
