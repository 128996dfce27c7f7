"""Performance cases of the package: what a program that serves Llama-family models does with it.

Two ways of use are covered.  A *runner* (``CudaTransformerRunner``) owns a model: prompts are fed, tokens generated
greedily, with the device sampler, or from logits that the host picks from, for one sequence or for several.  The
*backend* (``CudaB200Backend``, the ``ComputeBackend`` trait) is called op by op by hosts that keep their own forward
pass.  Shapes are those of ``yule_b200.synth`` (1.1B, 8B and 70B architectures); weights are random blocks whose
dequantised values have the spread of a trained model's (about 0.02), activations are N(0, 1).

A case is a dict: ``kind`` says which use it is, the other keys its sizes.  ``listed()`` holds the fixed ones, ``draw``
takes more from the same ranges.
"""

from __future__ import annotations

import dataclasses
import math

import numpy as np
import torch

from yule_b200 import CudaB200Backend, CudaTransformerRunner, DType, synth

MODELS = {"1b": synth.TINYLLAMA, "8b": synth.LLAMA3_8B, "70b": synth.LLAMA3_70B}

_backend = None


def backend() -> CudaB200Backend:
    """A program has one backend; all its buffers and runners live on it."""
    global _backend
    if _backend is None:
        _backend = CudaB200Backend(0)
    return _backend


# ── the cases ──────────────────────────────────────────────────────────────────────────────────


def listed() -> list[dict]:
    return [
        # A host with its own forward pass, one call per op: a token through four layers of the 1.1B shape after a
        # hundred tokens of context.  Small kernels; launches and calls count.
        {"name": "ops-1b", "kind": "ops", "model": "1b", "layers": 4, "fmt": "Q4_K", "pos": 100},
        # The smallest call: one matrix of the 1.1B model (its FFN-up projection) times one vector, read back.
        {"name": "matmul-q4k-1", "kind": "matmul", "fmt": "Q4_K", "rows": 5632, "cols": 2048, "batch": 1},
        # The down projection of the 8B model for four rows at once (a small batch, speculative tokens), 8-bit weights.
        {"name": "matmul-q8_0-4", "kind": "matmul", "fmt": "Q8_0", "rows": 4096, "cols": 14336, "batch": 4},
        # Decode attention alone over a full 4096-token cache, 8B head layout.
        {"name": "attention-4096", "kind": "attention", "model": "8b", "seq": 4096},
        # Greedy completion of a short prompt with the 1.1B model: latency of the token step.
        {"name": "generate-1b", "kind": "generate", "model": "1b", "layers": 22, "fmt": "Q4_K", "prompt": 32, "gen": 128},
        # A chat turn whose host picks from the logits itself, 8-bit weights: short prompt, then single steps.
        {"name": "chat-1b-q8_0", "kind": "chat", "model": "1b", "layers": 22, "fmt": "Q8_0", "prompt": 25, "gen": 32},
        # Sampled completion (default sampling parameters), 4-bit legacy format, few layers of the 8B shape with its
        # large vocabulary.
        {"name": "sampled-8b-q4_0", "kind": "sampled", "model": "8b", "layers": 8, "fmt": "Q4_0", "prompt": 60, "gen": 64},
        # A document of odd length through the 1.1B model: prompt processing, logits of its last token.
        {"name": "prompt-1b", "kind": "prompt", "model": "1b", "layers": 22, "fmt": "Q4_K", "prompt": 777},
        # Eight conversations served together by the 1.1B model: equal short prompts, greedy answers.
        {"name": "batch8-1b", "kind": "batch", "model": "1b", "layers": 22, "fmt": "Q4_K", "batch": 8, "prompt": 40, "gen": 40},
        # The full 8B model: a 2048-token prompt.
        {"name": "prompt-8b", "kind": "prompt", "model": "8b", "layers": 32, "fmt": "Q4_K", "prompt": 2048},
        # The full 8B model: greedy completion.
        {"name": "generate-8b", "kind": "generate", "model": "8b", "layers": 32, "fmt": "Q4_K", "prompt": 100, "gen": 64},
        # Layers of the 70B shape (a tenth of the model, to bound the set-up), thirty-two sequences together.
        {"name": "batch32-70b", "kind": "batch", "model": "70b", "layers": 8, "fmt": "Q4_K", "batch": 32, "prompt": 16, "gen": 20},
    ]


def _log(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    """One more case of the ranges above.  Runner cases bound layers x tokens so that none costs more than the largest
    listed one."""
    kind = rng.choice(["ops", "matmul", "attention", "generate", "chat", "sampled", "prompt", "batch"])
    fmt = rng.choice(["Q4_K", "Q4_K", "Q4_K", "Q6_K", "Q8_0", "Q4_0", "Q5_K"])
    if kind == "matmul":
        batch = rng.choice([1, 1, 2, 3, 4, 6, 8, 13, 16, 24, 32, _log(rng, 33, 300)])
        cols = 256 * _log(rng, 4, 56)
        rows = _log(rng, 1024, 32768 if batch <= 16 else 8192)
        return {"kind": kind, "fmt": fmt, "rows": rows, "cols": cols, "batch": batch}
    if kind == "attention":
        return {"kind": kind, "model": rng.choice(["1b", "8b", "70b"]), "seq": _log(rng, 60, 16000)}
    model = rng.choice(["1b", "1b", "8b", "8b", "70b"])
    if kind == "ops":
        return {"kind": kind, "model": model, "layers": rng.randint(1, 4), "fmt": fmt, "pos": _log(rng, 1, 1500)}
    layers = {"1b": rng.randint(8, 22), "8b": rng.randint(4, 16), "70b": rng.randint(2, 6)}[model]
    case = {"kind": kind, "model": model, "layers": layers, "fmt": fmt}
    if kind == "generate":
        case.update(prompt=_log(rng, 4, 500), gen=rng.randint(16, 100))
    elif kind == "chat":
        case.update(prompt=_log(rng, 4, 500), gen=rng.randint(8, 40))
    elif kind == "sampled":
        case.update(prompt=_log(rng, 4, 500), gen=rng.randint(16, 80))
    elif kind == "prompt":
        case.update(prompt=_log(rng, 17, 3000 if model == "1b" else 2000))
    else:
        case.update(batch=rng.choice([2, 3, 4, 5, 8, 12, 16, 20, 32, 48]), prompt=_log(rng, 4, 60), gen=rng.randint(16, 48))
    while work(case)["bytes"] > 2.5e11:
        case["gen"] = case["gen"] * 3 // 4
    return case


# ── inputs ─────────────────────────────────────────────────────────────────────────────────────


def _config(case: dict):
    cfg = MODELS[case["model"]]
    if case["kind"] in ("ops", "attention"):
        return dataclasses.replace(cfg, n_layers=case.get("layers", 1))
    # the context a program asks for: the whole of the model's for one sequence, what it needs for many
    ctx = cfg.max_seq_len if case["kind"] != "batch" else 256
    return dataclasses.replace(cfg, n_layers=case["layers"], max_seq_len=ctx)


def _formats(case: dict) -> dict:
    """Formats by role.  Q4_K files keep some matrices in Q6_K, the smaller the model the more of them."""
    dt = DType[case["fmt"]]
    roles = {"linear": dt, "down": dt, "output": dt}
    if dt == DType.Q4_K:
        if case["model"] == "1b":
            roles["down"] = DType.Q6_K
        if case["model"] != "70b":
            roles["output"] = DType.Q6_K
    return roles


def _format_of(name: str, roles: dict) -> DType:
    return roles["output"] if name == "output.weight" else roles["down"] if "ffn_down" in name else roles["linear"]


def _generator(seed: int) -> torch.Generator:
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _host(t: torch.Tensor) -> np.ndarray:
    """A tensor's bytes in pinned host memory, as a program that loads a model would stage them."""
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def _blocks(dt: DType, rows: int, cols: int, g: torch.Generator, row_spread: float = 0.0) -> torch.Tensor:
    """Random blocks of a format: uniform quants, scales such that the weights are centred with a spread of about 0.02.
    ``row_spread`` > 0 makes the rows of unequal size (log-normal)."""
    n, size = rows * cols // dt.block_size, dt.size_of_block
    b = torch.randint(-2 ** 63, 2 ** 63 - 1, ((n * size + 7) // 8,), generator=g, device="cuda", dtype=torch.int64)
    b = b.view(torch.uint8)[: n * size].view(n, size)
    jitter = torch.rand(n, generator=g, device="cuda") * 0.4 + 0.8
    if row_spread:
        jitter *= torch.exp(row_spread * torch.randn(rows, generator=g, device="cuda")).repeat_interleave(n // rows)

    def half(at: int, value: torch.Tensor) -> None:
        b[:, at:at + 2] = value.to(torch.float16).view(torch.uint8).view(n, 2)

    if dt in (DType.Q4_K, DType.Q5_K):
        # 6-bit scales in 32..63, each min equal to its scale, dmin = d times the middle quant
        b[:, 4:8] |= 0xA0
        b[:, 8:12] = b[:, 4:8]
        b[:, 12:16] = (b[:, 12:16] & 15) * 17
        middle, spread = (7.5, 4.6) if dt == DType.Q4_K else (15.5, 9.2)
        d = (jitter * (0.02 / (48 * spread))).to(torch.float16).float()
        half(0, d)
        half(2, d * middle)
    elif dt == DType.Q6_K:
        b[:, 192:208] = (b[:, 192:208] & 63) | 64
        half(208, jitter * (0.02 / (96 * 18.5)))
    elif dt == DType.Q8_0:
        half(0, jitter * (0.02 / 74))
    else:
        half(0, jitter * (0.02 / 4.6))
    return b.reshape(-1)


def _weights(cfg, roles: dict, g: torch.Generator) -> dict:
    """A model's tensors in host memory.  One layer's matrices serve all layers (each layer has its own device copy),
    so that making a large model is quick."""
    made, out = {}, {}
    for name, (rows, cols) in cfg.tensor_shapes().items():
        key = name.split(".", 2)[2] if name.startswith("blk.") else name
        if key not in made:
            dt = _format_of(name, roles)
            # a trained model's next-token distribution has few likely tokens: output rows of unequal size give that
            made[key] = (_host(_blocks(dt, rows, cols, g, 0.6 if key == "output.weight" else 0.0)), dt)
        out[name] = made[key]
    norm = _host((1 + 0.1 * torch.randn(cfg.dim, generator=g, device="cuda")).view(torch.uint8))
    for name in cfg.norm_names():
        out[name] = (norm, DType.F32)
    return out


class _Buffers:
    """Device buffers of a program, freed with it."""

    def __init__(self):
        self.b, self.handles = backend(), []

    def new(self, n_bytes: int):
        self.handles.append(self.b.allocate(n_bytes))
        return self.handles[-1]

    def up(self, array: np.ndarray):
        h = self.new(array.nbytes)
        self.b.copy_to_device(array, h)
        return h

    def matrix(self, dt: DType, rows: int, cols: int, g: torch.Generator):
        h = self.up(_host(_blocks(dt, rows, cols, g)))
        self.b.prepare_weights(h, dt, rows, cols)
        return h

    def __del__(self):
        for h in self.handles:
            self.b.free(h)


def prepare(case: dict, seed: int) -> dict:
    g = _generator(seed)
    kind = case["kind"]
    s = {"case": case, "b": backend()}
    if kind == "matmul":
        m = _Buffers()
        dt, rows, cols, n = DType[case["fmt"]], case["rows"], case["cols"], case["batch"]
        s.update(mem=m, dt=dt, w=m.matrix(dt, rows, cols, g), y=m.new(4 * n * rows),
                 x=m.up(_host(torch.randn(n * cols, generator=g, device="cuda"))),
                 out=torch.empty(n, rows, pin_memory=True).numpy())
        return s
    cfg = _config(case)
    s["cfg"] = cfg
    qdim, kvdim = cfg.n_heads * cfg.head_dim, cfg.n_kv_heads * cfg.head_dim
    if kind == "attention":
        m = _Buffers()
        rows = [torch.randn(n, generator=g, device="cuda") for n in (qdim, case["seq"] * kvdim, case["seq"] * kvdim)]
        q, k, v = (m.up(_host(r)) for r in rows)
        s.update(mem=m, q=q, k=k, v=v, y=m.new(4 * qdim), out=torch.empty(qdim, pin_memory=True).numpy())
        return s
    roles = _formats(case)
    if kind == "ops":
        m, dim, ff, seq = _Buffers(), cfg.dim, cfg.ff_dim, case["pos"] + 1
        layers = []
        for _ in range(cfg.n_layers):
            layer = {"attn_norm": m.up(_host(1 + 0.1 * torch.randn(dim, generator=g, device="cuda"))),
                     "ffn_norm": m.up(_host(1 + 0.1 * torch.randn(dim, generator=g, device="cuda")))}
            for name, rows, cols in (("q", qdim, dim), ("k", kvdim, dim), ("v", kvdim, dim), ("o", dim, qdim),
                                     ("gate", ff, dim), ("up", ff, dim), ("down", dim, ff)):
                layer[name] = m.matrix(roles["down" if name == "down" else "linear"], rows, cols, g)
            layer["k_cache"], layer["v_cache"] = (m.up(_host(torch.randn(seq * kvdim, generator=g, device="cuda")))
                                                  for _ in range(2))
            layers.append(layer)
        s.update(mem=m, layers=layers, roles=roles, x=_host(torch.randn(dim, generator=g, device="cuda")),
                 out=torch.empty(dim, pin_memory=True).numpy())
        for name, n in (("hidden", dim), ("normed", dim), ("qb", qdim), ("kb", kvdim), ("vb", kvdim), ("att", qdim),
                        ("proj", dim), ("gateb", ff), ("upb", ff)):
            s[name] = m.new(4 * n)
        return s
    weights = _weights(cfg, roles, g)
    # one sequence: the runner with the persistent token step where the model has one; several: the graph runner
    s["runner"] = CudaTransformerRunner(backend(), cfg, weights, fused=2 if kind in ("generate", "chat", "sampled", "prompt") else 1)
    n = case.get("batch", 1) * case["prompt"]
    tokens = torch.randint(0, cfg.vocab_size, (n,), generator=g, device="cuda").cpu().numpy().astype(np.uint32)
    s["prompt"] = tokens.reshape(case["batch"], -1) if kind == "batch" else tokens
    s["sample_seed"] = seed
    if kind == "chat":
        s["out"] = np.empty((case["gen"] + 1, cfg.vocab_size), np.float32)
    return s


# ── one pass ───────────────────────────────────────────────────────────────────────────────────


def _run_ops(s: dict) -> np.ndarray:
    b, cfg, lin, down = s["b"], s["cfg"], s["roles"]["linear"], s["roles"]["down"]
    dim, ff, hd, pos = cfg.dim, cfg.ff_dim, cfg.head_dim, s["case"]["pos"]
    qdim, kvdim = cfg.n_heads * hd, cfg.n_kv_heads * hd
    hidden, normed, q, k, v, att, proj, gate, up = (s[n] for n in ("hidden", "normed", "qb", "kb", "vb", "att", "proj", "gateb", "upb"))
    b.copy_to_device(s["x"], hidden)
    for L in s["layers"]:
        b.rms_norm(hidden, L["attn_norm"], normed, dim, cfg.norm_eps)
        b.quantized_matmul(L["q"], normed, q, qdim, dim, lin)
        b.quantized_matmul(L["k"], normed, k, kvdim, dim, lin)
        b.quantized_matmul(L["v"], normed, v, kvdim, dim, lin)
        b.rope(q, k, pos, hd, cfg.rope_freq_base, cfg.n_heads, cfg.n_kv_heads)
        b.copy_buffer_offset(k, L["k_cache"], 0, pos * kvdim * 4, kvdim * 4)
        b.copy_buffer_offset(v, L["v_cache"], 0, pos * kvdim * 4, kvdim * 4)
        b.multihead_attention(q, L["k_cache"], L["v_cache"], att, hd, pos + 1, cfg.n_heads, cfg.n_kv_heads, kvdim)
        b.quantized_matmul(L["o"], att, proj, dim, qdim, lin)
        b.add(hidden, proj, hidden, dim)
        b.rms_norm(hidden, L["ffn_norm"], normed, dim, cfg.norm_eps)
        b.quantized_matmul(L["gate"], normed, gate, ff, dim, lin)
        b.quantized_matmul(L["up"], normed, up, ff, dim, lin)
        b.element_mul(gate, up, gate, ff)
        b.quantized_matmul(L["down"], gate, proj, dim, ff, down)
        b.add(hidden, proj, hidden, dim)
    b.copy_from_device(hidden, s["out"])
    return s["out"]


def _pick(logits: np.ndarray) -> int:
    return int(np.argmax(logits))


def run(s: dict):
    case, b = s["case"], s["b"]
    kind = case["kind"]
    if kind == "ops":
        return _run_ops(s)
    if kind == "matmul":
        if case["batch"] == 1:
            b.quantized_matmul(s["w"], s["x"], s["y"], case["rows"], case["cols"], s["dt"])
        else:
            b.quantized_matmul_batched(s["w"], s["x"], s["y"], case["rows"], case["cols"], s["dt"], case["batch"])
        b.copy_from_device(s["y"], s["out"])
        return s["out"]
    if kind == "attention":
        cfg = s["cfg"]
        b.multihead_attention(s["q"], s["k"], s["v"], s["y"], cfg.head_dim, case["seq"], cfg.n_heads, cfg.n_kv_heads,
                              cfg.n_kv_heads * cfg.head_dim)
        b.copy_from_device(s["y"], s["out"])
        return s["out"]
    r = s["runner"]
    if kind == "batch":
        r.reset_batch()
        return r.generate_greedy_batch(s["prompt"], case["gen"])
    r.reset()
    if kind == "generate":
        return r.generate_greedy(s["prompt"], case["gen"])
    if kind == "sampled":
        return r.generate_sampled(s["prompt"], case["gen"], s["sample_seed"])
    if kind == "prompt":
        return r.prefill(s["prompt"])
    out = s["out"]
    out[0] = r.prefill(s["prompt"])
    for i in range(case["gen"]):
        r.decode_step(_pick(out[i]), out[i + 1])
    return out


# ── what a pass cannot do without ──────────────────────────────────────────────────────────────


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "matmul":
        rows, cols, n = case["rows"], case["cols"], case["batch"]
        return {"bytes": DType[case["fmt"]].tensor_bytes(rows, cols) + 4 * n * (rows + cols), "flops": 2 * rows * cols * n}
    cfg = _config(case)
    qdim, kvdim = cfg.n_heads * cfg.head_dim, cfg.n_kv_heads * cfg.head_dim
    if kind == "attention":
        return {"bytes": 8 * case["seq"] * kvdim + 8 * qdim, "flops": 4 * case["seq"] * qdim}
    roles = _formats(case)
    layer_bytes = layer_weights = 0
    for name, (rows, cols) in dataclasses.replace(cfg, n_layers=1).tensor_shapes().items():
        if name.startswith("blk."):
            layer_bytes += _format_of(name, roles).tensor_bytes(rows, cols)
            layer_weights += rows * cols
    body, params = cfg.n_layers * layer_bytes, cfg.n_layers * layer_weights
    head, head_params = roles["output"].tensor_bytes(cfg.vocab_size, cfg.dim), cfg.vocab_size * cfg.dim
    kv_row, att_pair = 8 * cfg.n_layers * kvdim, 4 * cfg.n_layers * qdim  # bytes of a K and V row, flops per (query, key)
    if kind == "ops":
        seq = case["pos"] + 1
        return {"bytes": body + kv_row * (seq + 1) + 8 * cfg.dim, "flops": 2 * params + att_pair * seq}
    n, p, gen = case.get("batch", 1), case["prompt"], case.get("gen", 0)
    # The prompt crosses the layers in one pass over the weights (its tokens are all known) and, like every later token,
    # needs one row of logits.  Each token that follows depends on the one before: the weights and the sequence's K and
    # V rows are read again.  Greedy and sampled generation feed their last token too.
    embed = n * (p + gen) * roles["linear"].tensor_bytes(1, cfg.dim)
    keys_read = n * (p + sum(p + i + 1 for i in range(gen)))
    keys_written = n * (p + gen)
    pairs = n * (p * (p + 1) // 2 + sum(p + i + 1 for i in range(gen)))
    logits_out = 4 * cfg.vocab_size * (1 if kind == "prompt" else gen + 1 if kind == "chat" else 0)
    return {"bytes": (1 + gen) * (body + head) + embed + kv_row * (keys_read + keys_written) + logits_out + 4 * n * (p + gen),
            "flops": 2 * n * (p + gen) * params + 2 * n * (1 + gen) * head_params + att_pair * pairs}


def tolerance(case: dict) -> dict:
    """fp32 results: sums of products formed in another order; a model's logits carry the differences of all its layers.
    Token streams are whole numbers: only a pick between logits (or a draw at a boundary) that agree to rounding may
    differ."""
    kind = case["kind"]
    if kind in ("generate", "sampled", "batch"):
        return {"rel": 0.0, "differ": 0.01}
    if kind in ("prompt", "chat"):
        return {"rel": 1e-4, "max": 1e-3}
    return {"rel": 1e-5, "max": 1e-4}
