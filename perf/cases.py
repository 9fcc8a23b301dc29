"""What the framework's users run, as cases that can be timed and checked: quantized linears, the attention block of a
GGUF LLaMA in prompts and in decoding, a whole LLaMA token step, and the layers of the sequence models (feed-forwards,
attention over a cache, delta rule, state-space scan, routed experts) as the models' lowerings emit them.

Every case is a compiled DeviceProgram (or a serving session over one) that is built in `prepare` and executed by `run`;
operands live in HBM, as they do between the ops of a model.  `exact` restates each case in 64-bit torch."""
import math

import numpy as np
import torch

from zgml_b200 import abi
from zgml_b200.backend import CudaBackend, DeviceBuffer, DeviceOp, DeviceProgram, ExternBuffer, QuantizedWeight, ResidentQuantizedWeight, seq_scratch_elems, seq_state_elems
from zgml_b200.host.llama import LINEARS, DeviceLlamaSession, LlamaConfig, LlamaWeights, linear_shapes, rope_tables

GGML_TYPE = {"q4_0": 2, "q8_0": 8}
BLOCK = 32
EPS = 1e-5
WDT = {"bf16": abi.W_BF16, "f32": abi.W_F32}

# What each listed case stands for:
LISTED = [
    # one decoded token's linears, batch 1, int4 blocks (the matvec shape every 8B-size LLaMA layer has); eight layers' worth of weights
    {"name": "decode_linears_q4_0", "kind": "linear", "fmt": "q4_0", "rows": 1, "inputs": 4096, "outputs": 4096, "layers": 8},
    # six sequences decoded together: the feed-forward's gate / up product
    {"name": "batch_linears_q8_0", "kind": "linear", "fmt": "q8_0", "rows": 6, "inputs": 4096, "outputs": 14336, "layers": 2},
    # a 2048-token prompt through one feed-forward linear of an 8B-size LLaMA
    {"name": "prefill_linear_q8_0", "kind": "linear", "fmt": "q8_0", "rows": 2048, "inputs": 4096, "outputs": 14336, "layers": 1},
    # the attention block (rotary, cache stores, attention, concatenation) of that prompt
    {"name": "llama_attention_prefill", "kind": "llama_attention", "tokens": 2048, "context": 0, "heads": 32, "kv_heads": 8, "head_dim": 128, "max_seq": 2048},
    # one token of a SmolLM-135M-shape model with 512 tokens behind it, host token in, host logits out: latency and launches
    {"name": "llama_token_step", "kind": "llama_step", "fmt": "q8_0", "layers": 30, "width": 576, "heads": 9, "kv_heads": 3, "ff": 1536, "vocab": 49152, "context": 512},
    # feed-forward sublayers of a sequence model, one token: a chain of small launches
    {"name": "ffn_decode_bf16", "kind": "ffn", "tokens": 1, "width": 2048, "ff": 4096, "layers": 4, "dtype": "bf16", "gated": True},
    # the same sublayer in a float32 session, a session's default chunk of a prompt
    {"name": "ffn_prefill_f32", "kind": "ffn", "tokens": 256, "width": 2048, "ff": 4096, "layers": 1, "dtype": "f32", "gated": True},
    # grouped-query attention of a 1024-token chunk that follows 1024 cached positions
    {"name": "cached_attention_prefill", "kind": "cached_attention", "tokens": 1024, "position": 1024, "heads": 16, "kv_heads": 4, "dk": 128, "dv": 128,
     "mask": "causal", "size": 0, "sink": False, "latent": False},
    # one token's latent attention (absorbed form) over 8192 cached positions
    {"name": "latent_attention_decode", "kind": "cached_attention", "tokens": 1, "position": 8192, "heads": 16, "kv_heads": 1, "dk": 576, "dv": 512,
     "mask": "causal", "size": 0, "sink": True, "latent": True},
    # delta-rule mixer of a 1024-token chunk, one decay per key channel
    {"name": "delta_rule_prefill", "kind": "delta_rule", "tokens": 1024, "heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "dtype": "bf16", "head_decay": False},
    # state-space mixer of a 1024-token chunk, and the token decoded after it
    {"name": "ssm_scan_prefill", "kind": "ssm", "tokens": 1024, "heads": 64, "groups": 1, "state": 128, "head_dim": 64, "dtype": "bf16"},
    # routed experts for a 1024-token chunk
    {"name": "moe_prefill_bf16", "kind": "moe", "tokens": 1024, "width": 2048, "ff": 2048, "experts": 16, "top": 2, "dtype": "bf16"},
]


def listed():
    return [dict(c) for c in LISTED]


def _log(rng, lo, hi, step=1):
    """A whole number spread over the logarithm of [lo, hi], a multiple of `step`."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5)))))
    return max(lo, min(hi, (v + step // 2) // step * step))


def draw(rng):
    kind = rng.choice(["linear", "linear", "llama_attention", "llama_step", "ffn", "ffn", "cached_attention", "cached_attention", "delta_rule", "ssm", "moe"])
    if kind == "linear":
        rows = rng.choice([1, rng.randint(2, 8), _log(rng, 9, 2048)])
        inputs, outputs = _log(rng, 512, 14336, 32), _log(rng, 512, 14336, 32)
        while inputs * outputs > 4096 * 14336:
            outputs = _log(rng, 512, outputs, 32)
        return {"kind": kind, "fmt": rng.choice(["q4_0", "q8_0", "i8_f32"]), "rows": rows, "inputs": inputs, "outputs": outputs, "layers": rng.randint(1, 4) if rows <= 8 else 1}
    if kind == "llama_attention":
        head_dim, kv = rng.choice([64, 128]), rng.choice([2, 3, 4, 8])
        tokens, context = rng.choice([1, _log(rng, 16, 1536)]), rng.randint(0, 512)
        return {"kind": kind, "tokens": tokens, "context": context, "heads": kv * rng.choice([1, 2, 4]), "kv_heads": kv, "head_dim": head_dim, "max_seq": 2048}
    if kind == "llama_step":
        kv = rng.choice([1, 2, 4])
        heads = kv * rng.choice([1, 2, 3])
        return {"kind": kind, "fmt": rng.choice(["q4_0", "q8_0"]), "layers": rng.randint(4, 12), "width": 64 * heads, "heads": heads, "kv_heads": kv,
                "ff": _log(rng, 256, 2048, 32), "vocab": _log(rng, 4096, 32768, 32), "context": rng.randint(16, 256)}
    if kind == "ffn":
        dtype = rng.choice(["bf16", "bf16", "f32"])
        tokens = rng.choice([1, rng.randint(2, 8), _log(rng, 9, 1024 if dtype == "bf16" else 384)])
        return {"kind": kind, "tokens": tokens, "width": _log(rng, 256, 3072, 8), "ff": _log(rng, 512, 6144, 8), "layers": rng.randint(2, 4) if tokens <= 8 else 1,
                "dtype": dtype, "gated": rng.random() < 0.5}
    if kind == "cached_attention":
        mask = rng.choice(["causal", "causal", "window"])
        size = _log(rng, 64, 1024) if mask == "window" else 0
        if rng.random() < 0.25:       # a latent in its absorbed form: decoding and short steps
            return {"kind": kind, "tokens": rng.choice([1, rng.randint(2, 64)]), "position": _log(rng, 64, 8192), "heads": rng.choice([4, 8, 16]), "kv_heads": 1,
                    "dk": 320, "dv": 256, "mask": mask, "size": size, "sink": rng.random() < 0.5, "latent": True}
        kv, dim = rng.choice([1, 2, 4]), rng.choice([32, 64, 96, 128])
        return {"kind": kind, "tokens": rng.choice([1, _log(rng, 2, 1024)]), "position": rng.choice([0, _log(rng, 16, 4096)]), "heads": kv * rng.choice([1, 2, 4]), "kv_heads": kv,
                "dk": dim + rng.choice([0, 0, 32]), "dv": dim, "mask": mask, "size": size, "sink": rng.random() < 0.3, "latent": False}
    if kind == "delta_rule":
        kv, dim = rng.choice([1, 2, 4]), rng.choice([32, 64, 96, 128])
        return {"kind": kind, "tokens": rng.choice([1, _log(rng, 2, 1024)]), "heads": kv * rng.choice([1, 2, 4]), "kv_heads": kv, "dim": dim, "vdim": rng.choice([dim, 64, 128]),
                "dtype": rng.choice(["bf16", "f32"]), "head_decay": rng.random() < 0.4}
    if kind == "ssm":
        groups = rng.choice([1, 2])
        return {"kind": kind, "tokens": rng.choice([1, _log(rng, 2, 1024)]), "heads": groups * rng.choice([4, 8, 16, 32]), "groups": groups, "state": rng.choice([32, 64, 128]),
                "head_dim": rng.choice([32, 64, 128]), "dtype": rng.choice(["bf16", "f32"])}
    return {"kind": kind, "tokens": rng.choice([1, rng.randint(2, 8), _log(rng, 9, 1024)]), "width": _log(rng, 256, 2048, 8), "ff": _log(rng, 256, 2048, 8),
            "experts": rng.choice([4, 8, 16]), "top": rng.choice([1, 2]), "dtype": "bf16"}


# ── inputs: made on the GPU from the seed alone, the same tensors for `prepare` and `exact` ──────────────────────────
class _Random:
    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(0x5EED + seed)

    def normal(self, *shape, scale=1.0):
        return torch.randn(*shape, generator=self.g, device="cuda", dtype=torch.float32) * scale

    def uniform(self, *shape, lo=0.0, hi=1.0):
        return torch.rand(*shape, generator=self.g, device="cuda", dtype=torch.float32) * (hi - lo) + lo

    def integers(self, lo, hi, *shape):
        return torch.randint(lo, hi, shape, generator=self.g, device="cuda")

    def weight(self, n, k, dtype):
        """[n, k] linear weight of unit-variance products, in the values the session's weight format holds."""
        w = self.normal(n, k, scale=k ** -0.5)
        return w.to(torch.bfloat16) if dtype == "bf16" else w


def _quantized(r, fmt, K, N):
    """(whole numbers [K, N / 32, 32], scales [K, N / 32]) of a random [K, N] weight in a block format."""
    q = r.integers(-8, 8, K, N // BLOCK, BLOCK) if fmt == "q4_0" else r.integers(-127, 128, K, N // BLOCK, BLOCK)
    s = r.uniform(K, N // BLOCK, lo=0.5, hi=1.0) * (math.sqrt(6.0 / K) / (7 if fmt == "q4_0" else 127))
    return q.to(torch.int8), s if fmt == "i8_f32" else s.to(torch.float16).float()


def _upload(be, fmt, q, s):
    """The weight as a model file holds it (GGUF blocks), or as zgml's own quantizer leaves it (i8 + f32 scales)."""
    K, nb, _ = q.shape
    if fmt == "i8_f32":
        return QuantizedWeight.upload(be, q.reshape(-1).cpu().numpy(), s.reshape(-1).cpu().numpy(), K, nb * BLOCK)
    head = s.to(torch.float16).reshape(-1, 1).view(torch.uint8)
    if fmt == "q8_0":
        body = q.reshape(-1, BLOCK).view(torch.uint8)
    else:
        u = (q.reshape(-1, BLOCK) + 8).to(torch.uint8)
        body = u[:, 0::2] | (u[:, 1::2] << 4)
    return QuantizedWeight.from_gguf_blocks(be, torch.cat([head, body], 1).reshape(-1).cpu().numpy(), GGML_TYPE[fmt], K, nb * BLOCK)


def _dense(q, s):
    return (q.double() * s.double()[..., None]).reshape(q.shape[0], -1)


# ── programs ─────────────────────────────────────────────────────────────────────────────────────────────────────────
_BACKEND = []


def _backend():
    """The one backend a serving process keeps."""
    if not _BACKEND:
        _BACKEND.append(CudaBackend(0))
    return _BACKEND[0]


class _DeviceArray:
    """Device memory as torch reads it; a tensor over it keeps `owner`, which frees the memory, alive."""

    def __init__(self, ptr, n, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": (int(n),), "typestr": "<f4", "version": 3}


def _tensor(owner, ptr, n, *shape):
    return torch.as_tensor(_DeviceArray(ptr, n, owner), device="cuda").view(*shape)


class _Program:
    """A compiled program with its operands, and views of the buffers it leaves results in."""

    def __init__(self):
        self.be, self.sizes, self.ops, self.externs, self.weights, self.owned, self.handle = _backend(), [], [], [], [], [], None

    def buf(self, n):
        self.sizes.append(max(int(n), 1))
        return len(self.sizes) - 1

    def ext(self, b):
        self.sizes.append(b.elems)
        self.externs.append(ExternBuffer(len(self.sizes) - 1, b))
        return len(self.sizes) - 1

    def dense(self, *tensors):
        """(buffer, element offsets) of weights or state laid back to back, each at a 16-byte boundary, in one device buffer."""
        offs, flat, n = [], [], 0
        for t in tensors:
            offs.append(n)
            t = t.reshape(-1)
            pad = -t.numel() % 8
            flat.append(torch.cat([t, t.new_zeros(pad)]) if pad else t)
            n += flat[-1].numel()
        flat = torch.cat(flat)
        b = DeviceBuffer(self.be, flat.numel() * flat.element_size(), zero=False)
        self.owned.append(b)
        _tensor(b, b.ptr, b.elems, -1).view(flat.dtype).copy_(flat)
        return b, offs

    def compile(self):
        self.handle = self.be.compile_program(DeviceProgram(self.ops, self.sizes, [], [ResidentQuantizedWeight(w) for w in self.weights], self.externs))
        if self.handle is None:
            raise RuntimeError("the program did not compile")
        return self

    def tensor(self, b, *shape):
        return _tensor(self, self.be.lib.zg_cuda_program_buffer(self.handle.ptr, b), self.sizes[b], *shape)

    def ctl(self, b, words):
        c = torch.zeros(self.sizes[b], dtype=torch.int32, device="cuda")
        c[:len(words)] = torch.tensor(words, dtype=torch.int32)
        self.tensor(b, -1).view(torch.int32).copy_(c)

    def execute(self):
        self.be.lib.zg_cuda_execute_device(self.be.ctx, self.handle.ptr)

    def __del__(self):
        if self.handle is not None:
            self.be.sync()
            self.be.free_program(self.handle)
        for w in self.weights:
            w.free()
        for b in self.owned:
            b.free()


class _State:
    def __init__(self, programs, outputs):
        self.programs, self.outputs = programs, outputs


def prepare(case, seed):
    state = globals()["_prepare_" + case["kind"]](case, _Random(seed))
    torch.cuda.synchronize()
    return state


def run(state):
    if isinstance(state, _Step):
        return state.session.execute_at([state.token], state.context)
    for p in state.programs:
        p.execute()
    return state.outputs


def exact(case, seed):
    return globals()["_exact_" + case["kind"]](case, _Random(seed))


def work(case):
    return globals()["_work_" + case["kind"]](case)


def tolerance(case):
    """About four times the error against 64 bits that the path shows at these sizes."""
    if case["kind"] == "linear":
        # up to 8 rows: a 23-bit grid for the scaled activations; more rows: products of bfloat16 pairs
        return {"rel": 2.5e-6 if case["rows"] <= 8 else 6e-5}
    if case["kind"] == "llama_step":
        return {"rel": 2e-5}
    if case["kind"] in ("ffn", "moe") and case["dtype"] == "bf16":
        # many rows of bfloat16 weights round their activations once per product; few rows are summed in f32
        rows = case["tokens"] * case.get("top", 1)
        return {"rel": 1.2e-2 if rows > (16 if case["kind"] == "moe" else 8) else 4e-6}
    return {"rel": 5e-6}


# ── quantized linears ────────────────────────────────────────────────────────────────────────────────────────────────
def _inputs_linear(case, r):
    K, N = case["inputs"], case["outputs"]
    ws = [_quantized(r, case["fmt"], K, N) for _ in range(case["layers"])]
    return ws, r.normal(case["rows"], K)


def _prepare_linear(case, r):
    M, K, N = case["rows"], case["inputs"], case["outputs"]
    ws, x = _inputs_linear(case, r)
    p = _Program()
    p.weights = [_upload(p.be, case["fmt"], q, s) for q, s in ws]
    src, dst = p.buf(M * K), [p.buf(M * N) for _ in ws]
    p.ops = [DeviceOp.qmatmul(d, src, i, M, N, K) for i, d in enumerate(dst)]
    p.compile()
    p.tensor(src, M, K).copy_(x)
    return _State([p], [p.tensor(d, M, N) for d in dst])


def _exact_linear(case, r):
    ws, x = _inputs_linear(case, r)
    return [x.double() @ _dense(q, s) for q, s in ws]


def _work_linear(case):
    M, K, N, n = case["rows"], case["inputs"], case["outputs"], case["layers"]
    return {"bytes": n * (K * N // BLOCK * {"q4_0": 18, "q8_0": 34, "i8_f32": 36}[case["fmt"]] + 4 * M * N) + 4 * M * K, "flops": 2 * n * M * K * N}


# ── the attention block of a LLaMA layer ─────────────────────────────────────────────────────────────────────────────
def _inputs_llama_attention(case, r):
    T, H, G, d, S, p0 = (case[k] for k in ("tokens", "heads", "kv_heads", "head_dim", "max_seq", "context"))
    q, k, v = r.normal(T, H, d, scale=1.5), r.normal(T, G, d, scale=1.5), r.normal(T, G, d)
    kc, vc = r.normal(G, S, d, scale=1.5), r.normal(G, S, d)
    kc[:, p0:], vc[:, p0:] = 0.0, 0.0
    angle = torch.arange(p0, p0 + T, device="cuda", dtype=torch.float64)[:, None] * 1e4 ** (-2.0 * torch.arange(d // 2, device="cuda", dtype=torch.float64) / d)
    return q, k, v, kc, vc, angle.cos().float(), angle.sin().float()


def _prepare_llama_attention(case, r):
    T, H, G, d, S, p0 = (case[k] for k in ("tokens", "heads", "kv_heads", "head_dim", "max_seq", "context"))
    q, k, v, kc, vc, cos, sin = _inputs_llama_attention(case, r)
    p = _Program()
    bq, bk, bv, bkc, bvc, cs, mask, cat = p.buf(T * H * d), p.buf(T * G * d), p.buf(T * G * d), p.buf(G * S * d), p.buf(G * S * d), p.buf(2 * d * T), p.buf(S * T), p.buf(T * H * d)
    for g in range(G):
        kr, base = p.buf(d * T), g * S * d
        p.ops.append(DeviceOp.rope(kr, bk, cs, d // 2, T, g * d, 0, 0, 1, G * d, 2 * d))
        p.ops.append(DeviceOp.slice_assign(bkc, kr, d, T, base, base + p0 * d, 1, d, 0, 1, d, d))
        p.ops.append(DeviceOp.slice_assign(bvc, bv, d, T, base, base + p0 * d, 1, d, g * d, 1, G * d, d))
    for h in range(H):
        qr, out, base = p.buf(d * T), p.buf(d * T), h // (H // G) * S * d
        p.ops.append(DeviceOp.rope(qr, bq, cs, d // 2, T, h * d, 0, 0, 1, H * d, 2 * d))
        p.ops.append(DeviceOp.attention(out, qr, bkc, bvc, mask, True, d, T, p0 + T, float(np.float32(1) / np.sqrt(np.float32(d))), 0, base, base, 0, 0,
                                        1, d, 1, d, 1, d, 1, S, 1, d))
        p.ops.append(DeviceOp.slice_assign(cat, out, d, T, 0, h * d, 1, H * d, 0, 1, d, 0))
    p.compile()
    for b, t in ((bq, q), (bk, k), (bv, v), (bkc, kc), (bvc, vc), (cs, torch.cat([cos, sin, cos, sin], 1))):
        p.tensor(b, -1).copy_(t.reshape(-1))
    j, t = torch.arange(S, device="cuda")[None, :], torch.arange(T, device="cuda")[:, None]
    p.tensor(mask, T, S).copy_(torch.where(j <= p0 + t, 0.0, -math.inf))
    return _State([p], [p.tensor(cat, T, H, d), p.tensor(bkc, G, S, d), p.tensor(bvc, G, S, d)])


def _turn(x, cos, sin):
    a, b = x.double().chunk(2, -1)
    c, s = cos.double()[:, None], sin.double()[:, None]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _exact_llama_attention(case, r):
    T, H, G, d, S, p0 = (case[k] for k in ("tokens", "heads", "kv_heads", "head_dim", "max_seq", "context"))
    q, k, v, kc, vc, cos, sin = _inputs_llama_attention(case, r)
    q, kc, vc = _turn(q, cos, sin), kc.double(), vc.double()
    kc[:, p0:p0 + T], vc[:, p0:p0 + T] = _turn(k, cos, sin).transpose(0, 1), v.double().transpose(0, 1)
    out = torch.empty(T, H, d, dtype=torch.float64, device="cuda")
    dead = torch.arange(p0 + T, device="cuda")[None, :] > p0 + torch.arange(T, device="cuda")[:, None]
    for h in range(H):
        s = (q[:, h] @ kc[h // (H // G), :p0 + T].T * d ** -0.5).masked_fill(dead, -math.inf)
        out[:, h] = s.softmax(-1) @ vc[h // (H // G), :p0 + T]
    return [out, kc, vc]


def _pairs(T, p0, window):
    """(query, visible key) pairs of T tokens from position p0."""
    p = np.arange(p0, p0 + T)
    return int(np.minimum(p + 1, window).sum()) if window else int((p + 1).sum())


def _work_llama_attention(case):
    T, H, G, d, p0 = (case[k] for k in ("tokens", "heads", "kv_heads", "head_dim", "context"))
    return {"bytes": 4 * d * (2 * T * H + 2 * G * (p0 + T) + 4 * T * G), "flops": 4 * d * H * _pairs(T, p0, 0)}


# ── a whole LLaMA token ──────────────────────────────────────────────────────────────────────────────────────────────
class _Step:
    def __init__(self, weights, session, token, context):
        self.weights, self.session, self.token, self.context = weights, session, token, context

    def __del__(self):
        self.session.close()
        for w in self.weights:
            w.free()


def _llama_config(case):
    return LlamaConfig(case["vocab"], case["width"], case["layers"], case["heads"], case["kv_heads"], case["ff"], case["context"] + 64, EPS, 1e4, True)


def _inputs_llama_step(case, r):
    cfg = _llama_config(case)
    layers = [{n: _quantized(r, case["fmt"], *linear_shapes(cfg)[n]) for n in LINEARS} for _ in range(cfg.n_layers)]
    norms = r.uniform(2 * cfg.n_layers + 1, cfg.d_model, lo=0.8, hi=1.2)
    embed = r.uniform(cfg.vocab_size, cfg.d_model, lo=-0.05, hi=0.05)
    return cfg, layers, norms, embed, r.integers(0, cfg.vocab_size, case["context"] + 1)


def _prepare_llama_step(case, r):
    cfg, layers, norms, embed, tokens = _inputs_llama_step(case, r)
    be, handles, up = _backend(), [], []
    for L in layers:
        up.append({})
        for n, (q, s) in L.items():
            handles.append(_upload(be, case["fmt"], q, s))
            up[-1][n] = ResidentQuantizedWeight(handles[-1])
    norms, tokens = norms.cpu().numpy(), tokens.tolist()
    w = LlamaWeights(cfg, embed.cpu().numpy(), up, list(norms[:cfg.n_layers]), list(norms[cfg.n_layers:-1]), norms[-1])
    session = DeviceLlamaSession(be, cfg, w, 1)
    for t in tokens[:-1]:
        session.step(t)
    return _Step(handles, session, tokens[-1], case["context"])


def _exact_llama_step(case, r):
    cfg, layers, norms, embed, tokens = _inputs_llama_step(case, r)
    n, H, G, d = case["context"] + 1, cfg.n_heads, cfg.n_kv_heads, cfg.d_head
    # a column of the session's rotary table is [cos cos sin sin]; the ROPE op takes its second quarter as the sine
    table = np.concatenate([t[:n] for t in rope_tables(cfg)], 1)
    cos, sin = (torch.from_numpy(table[:, i * d // 2:(i + 1) * d // 2]).cuda() for i in (0, 1))
    rms = lambda x, w: x * (x.square().mean(-1, keepdim=True) + EPS).rsqrt() * w.double()  # noqa: E731
    dead = torch.ones(n, n, dtype=torch.bool, device="cuda").triu(1)
    x = embed[tokens].double()
    for i, L in enumerate(layers):
        W = {k: _dense(*v) for k, v in L.items()}
        h = rms(x, norms[i])
        q, k, v = _turn((h @ W["wq"]).view(n, H, d), cos, sin), _turn((h @ W["wk"]).view(n, G, d), cos, sin), (h @ W["wv"]).view(n, G, d)
        k, v = k.repeat_interleave(H // G, 1), v.repeat_interleave(H // G, 1)
        s = (torch.einsum("qhd,khd->hqk", q, k) * d ** -0.5).masked_fill(dead, -math.inf).softmax(-1)
        x = x + torch.einsum("hqk,khd->qhd", s, v).reshape(n, -1) @ W["wo"]
        h = rms(x, norms[cfg.n_layers + i])
        x = x + (torch.nn.functional.silu(h @ W["w_gate"]) * (h @ W["w_up"])) @ W["w_down"]
    return (rms(x[-1:], norms[-1]) @ embed.double().T).reshape(-1)


def _work_llama_step(case):
    cfg = _llama_config(case)
    n = case["layers"] * sum(k * m for k, m in linear_shapes(cfg).values())
    cache = 2 * case["layers"] * cfg.kv_dim * (case["context"] + 1)
    return {"bytes": n // BLOCK * {"q4_0": 18, "q8_0": 34}[case["fmt"]] + 4 * cache + 4 * cfg.vocab_size * (cfg.d_model + 1),
            "flops": 2 * n + 2 * cache * (cfg.n_heads // cfg.n_kv_heads) + 2 * cfg.vocab_size * cfg.d_model}


# ── feed-forward sublayers of the sequence models ────────────────────────────────────────────────────────────────────
def _inputs_ffn(case, r):
    T, D, F = case["tokens"], case["width"], case["ff"]
    layers = []
    for _ in range(case["layers"]):
        w = r.uniform(D, lo=0.8, hi=1.2)
        layers.append((w.to(torch.bfloat16) if case["dtype"] == "bf16" else w, r.weight(F * (2 if case["gated"] else 1), D, case["dtype"]), r.weight(D, F, case["dtype"])))
    return layers, r.normal(T, D)


def _prepare_ffn(case, r):
    T, D, F, wdt = case["tokens"], case["width"], case["ff"], WDT[case["dtype"]]
    layers, x = _inputs_ffn(case, r)
    p = _Program()
    src, h, u, y = p.buf(T * D), p.buf(T * D), p.buf(T * F), p.buf(T * D)
    arenas = [p.dense(*L) for L in layers]
    ws = [p.ext(b) for b, _ in arenas]
    p.ops.append(DeviceOp.norm(h, src, ws[0], arenas[0][1][0], T, D, EPS, wdt, kind="rms"))
    x_in = src
    for i in range(len(layers)):
        o = arenas[i][1]
        act = dict(act="silu", pairs=True) if case["gated"] else dict(act="relu2")
        p.ops.append(DeviceOp.linear(u, h, ws[i], o[1], T, F, D, wdt, **act))
        p.ops.append(DeviceOp.linear(y, u, ws[i], o[2], T, D, F, wdt))
        x_out = p.buf(T * D)
        then = {} if i + 1 == len(layers) else dict(then=h, then_w=ws[i + 1], then_w_off=arenas[i + 1][1][0], then_kind="rms")
        p.ops.append(DeviceOp.norm(x_out, y, None, 0, T, D, EPS, wdt, kind="none", res=x_in, **then))
        x_in = x_out
    p.compile()
    p.tensor(src, T, D).copy_(x)
    return _State([p], p.tensor(x_in, T, D))


def _exact_ffn(case, r):
    layers, x = _inputs_ffn(case, r)
    x = x.double()
    for w, up, down in layers:
        h = x * (x.square().mean(-1, keepdim=True) + EPS).rsqrt() * w.double()
        z = h @ up.double().T
        u = torch.nn.functional.silu(z[:, 0::2]) * z[:, 1::2] if case["gated"] else z.relu().square()
        x = x + u @ down.double().T
    return x


def _work_ffn(case):
    T, D, F, n = case["tokens"], case["width"], case["ff"], case["layers"]
    params = n * D * F * (3 if case["gated"] else 2)
    return {"bytes": params * (2 if case["dtype"] == "bf16" else 4) + 8 * T * D, "flops": 2 * T * params}


# ── attention over a per-sequence cache ──────────────────────────────────────────────────────────────────────────────
def _rows(case):
    """Cached positions a sequence has room for: all of them, or a ring as long as the window and the step need."""
    n = case["position"] + case["tokens"]
    return min(n, case["size"] - 1 + case["tokens"]) if case["mask"] == "window" else n


def _inputs_cached_attention(case, r):
    T, H, G, dk, dv = (case[k] for k in ("tokens", "heads", "kv_heads", "dk", "dv"))
    width = dk if case["latent"] else G * (dk + dv)
    R = _rows(case)
    cache, rows, q, sink = r.normal(R, width), r.normal(T, width), r.normal(T, H * dk, scale=2.0 if not case["latent"] else 1.0), r.normal(H)
    kept = min(R, case["position"])       # rows of earlier positions; the others are still empty
    if kept < R:
        cache[[(case["position"] + i) % R for i in range(R - kept)]] = 0.0
    return cache, rows, q, sink


def _prepare_cached_attention(case, r):
    T, H, G, dk, dv, p0 = (case[k] for k in ("tokens", "heads", "kv_heads", "dk", "dv", "position"))
    cache, rows, q, sink = _inputs_cached_attention(case, r)
    R, width = cache.shape
    p = _Program()
    rs = H * dk + width
    proj, ctl, out = p.buf(T * rs), p.buf(abi.CTL_IDS + T), p.buf(T * H * dv)
    kept, _ = p.dense(cache)
    c = p.ext(kept)
    p.ops.append(DeviceOp.cache_append(c, proj, ctl, H * dk, 0, T, width, rs, width, R))
    sinks = {} if not case["sink"] else dict(sink=p.ext(p.dense(sink)[0]), sink_off=0, sink_wdt=abi.W_F32)
    p.ops.append(DeviceOp.cached_attention(out, proj, c, c, ctl, 0, 0, 0 if case["latent"] else G * dk, T, H, G, 1, dk, dv, rs, width, width, R, dk ** -0.5,
                                           mask=case["mask"], mask_size=case["size"], **sinks))
    p.compile()
    p.tensor(proj, T, rs).copy_(torch.cat([q, rows], 1))
    p.ctl(ctl, [p0])
    return _State([p], [p.tensor(out, T, H, dv), _tensor(p, kept.ptr, R * width, R, width)])


def _exact_cached_attention(case, r):
    T, H, G, dk, dv, p0 = (case[k] for k in ("tokens", "heads", "kv_heads", "dk", "dv", "position"))
    cache, rows, q, sink = _inputs_cached_attention(case, r)
    R = cache.shape[0]
    cache = cache.double()
    pos = torch.arange(p0, p0 + T, device="cuda")
    cache[pos % R] = rows.double()
    first = max(0, p0 - case["size"] + 1) if case["mask"] == "window" else 0
    j = torch.arange(first, p0 + T, device="cuda")
    seen = j[None, :] <= pos[:, None]
    if case["mask"] == "window":
        seen &= j[None, :] > pos[:, None] - case["size"]
    keys = cache[j % R]
    out = torch.empty(T, H, dv, dtype=torch.float64, device="cuda")
    for h in range(H):
        g = h // (H // G)
        k = keys[:, g * dk:(g + 1) * dk]
        v = keys[:, :dv] if case["latent"] else keys[:, G * dk + g * dv:G * dk + (g + 1) * dv]
        s = (q[:, h * dk:(h + 1) * dk].double() @ k.T * dk ** -0.5).masked_fill(~seen, -math.inf)
        if case["sink"]:
            s = torch.cat([s, sink[h].double().expand(T, 1)], 1)
        out[:, h] = s.softmax(-1)[:, :len(j)] @ v
    return [out, cache]


def _work_cached_attention(case):
    T, H, G, dk, dv, p0 = (case[k] for k in ("tokens", "heads", "kv_heads", "dk", "dv", "position"))
    window = case["size"] if case["mask"] == "window" else 0
    width = dk if case["latent"] else G * (dk + dv)
    keys = min(p0 + T, window - 1 + T) if window else p0 + T
    return {"bytes": 4 * (keys * width + 2 * T * width + T * H * (dk + dv)), "flops": 2 * (dk + dv) * H * _pairs(T, p0, window)}


# ── delta rule ───────────────────────────────────────────────────────────────────────────────────────────────────────
def _inputs_delta_rule(case, r):
    T, H, G, d, dv = (case[k] for k in ("tokens", "heads", "kv_heads", "dim", "vdim"))
    nd = H if case["head_decay"] else H * d
    qkv, beta, a, gate = r.normal(T, 2 * G * d + H * dv), r.normal(T, H), r.normal(T, nd), r.normal(T, H * dv)
    a_log, dt_bias, norm = r.uniform(H, lo=-1.0, hi=1.0), r.normal(nd, scale=0.5) - 3.0, r.uniform(dv, lo=0.8, hi=1.2)
    if case["dtype"] == "bf16":
        a_log, dt_bias, norm = (t.to(torch.bfloat16) for t in (a_log, dt_bias, norm))
    return qkv, beta, a, gate, a_log, dt_bias, norm, r.normal(H, d, dv, scale=0.2)


def _prepare_delta_rule(case, r):
    T, H, G, d, dv = (case[k] for k in ("tokens", "heads", "kv_heads", "dim", "vdim"))
    qkv, beta, a, gate, a_log, dt_bias, norm, S = _inputs_delta_rule(case, r)
    p = _Program()
    ins = [p.buf(t.numel()) for t in (qkv, beta, a, gate)]
    out, ctl = p.buf(T * H * dv), p.buf(abi.CTL_IDS + T)
    w, o = p.dense(a_log, dt_bias, norm)
    kept, _ = p.dense(S)
    p.ops.append(DeviceOp.delta_rule(out, *ins, p.ext(w), p.ext(kept), ctl, 0, G * d, 2 * G * d, 0, o[0], o[1], o[2], T, H, G, d, dv, qkv.shape[1], H, a.shape[1], H * dv,
                                     WDT[case["dtype"]], EPS, 1e-6, d ** -0.5, head_decay=case["head_decay"]))
    p.compile()
    for b, t in zip(ins, (qkv, beta, a, gate)):
        p.tensor(b, -1).copy_(t.reshape(-1))
    return _State([p], [p.tensor(out, T, H, dv), _tensor(p, kept.ptr, H * d * dv, H, d, dv)])


def _exact_delta_rule(case, r):
    T, H, G, d, dv = (case[k] for k in ("tokens", "heads", "kv_heads", "dim", "vdim"))
    qkv, beta, a, gate, a_log, dt_bias, norm, S = (t.double() for t in _inputs_delta_rule(case, r))
    unit = lambda x: x * (x.square().sum(-1, keepdim=True) + 1e-6).rsqrt()  # noqa: E731
    q = (unit(qkv[:, :G * d].view(T, G, d)) * d ** -0.5).repeat_interleave(H // G, 1)
    k = unit(qkv[:, G * d:2 * G * d].view(T, G, d)).repeat_interleave(H // G, 1)
    v, b = qkv[:, 2 * G * d:].view(T, H, dv), beta.sigmoid()
    z = torch.nn.functional.softplus(a + dt_bias).view(T, H, -1)
    g = torch.exp(-a_log.exp()[None, :, None] * z).expand(T, H, d)
    out = torch.empty(T, H, dv, dtype=torch.float64, device="cuda")
    for t in range(T):
        S = S * g[t][:, :, None]
        u = b[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None, :]
        out[t] = torch.einsum("hkv,hk->hv", S, q[t])
    out = out * (out.square().mean(-1, keepdim=True) + EPS).rsqrt() * norm * gate.view(T, H, dv).sigmoid()
    return [out, S]


def _work_delta_rule(case):
    T, H, G, d, dv = (case[k] for k in ("tokens", "heads", "kv_heads", "dim", "vdim"))
    return {"bytes": 4 * (T * (2 * G * d + 3 * H * dv + H + H * (1 if case["head_decay"] else d)) + 2 * H * d * dv), "flops": 7 * T * H * d * dv}


# ── state-space scan ─────────────────────────────────────────────────────────────────────────────────────────────────
def _inputs_ssm(case, r):
    T, H, G, N, P = (case[k] for k in ("tokens", "heads", "groups", "state", "head_dim"))
    xbc, dt = r.normal(T + 1, H * P + 2 * G * N, scale=0.6), r.normal(T + 1, H)
    a_log, bias, skip = torch.log(1.0 + 15.0 * r.uniform(H)), r.uniform(H, lo=-5.0, hi=-1.0), r.uniform(H, lo=0.5, hi=1.5)
    if case["dtype"] == "bf16":
        a_log, bias, skip = (t.to(torch.bfloat16) for t in (a_log, bias, skip))
    return xbc, dt, a_log, bias, skip


def _prepare_ssm(case, r):
    T, H, G, N, P = (case[k] for k in ("tokens", "heads", "groups", "state", "head_dim"))
    xbc, dt, *w = _inputs_ssm(case, r)
    programs, outs, kept, first = [], [], None, 0
    for n in (T, 1):              # the chunk, and the token decoded from the state it leaves
        p = _Program()
        bx, bd, out, ctl = p.buf(n * xbc.shape[1]), p.buf(n * H), p.buf(n * H * P), p.buf(abi.CTL_IDS + n)
        arena, o = p.dense(*w)
        wb, args = p.ext(arena), (0, H * P, H * P + G * N, 0, o[0], o[1], o[2], n, H, G, N, P, xbc.shape[1], H, WDT[case["dtype"]])
        if kept is None:
            kept = DeviceBuffer(p.be, 4 * seq_state_elems(DeviceOp.ssm_scan(out, bx, bd, wb, 0, ctl, *args)))
            p.owned.append(kept)
        p.ops.append(DeviceOp.ssm_scan(out, bx, bd, wb, p.ext(kept), ctl, *args))
        p.compile()
        p.tensor(bx, -1).copy_(xbc[first:first + n].reshape(-1))
        p.tensor(bd, -1).copy_(dt[first:first + n].reshape(-1))
        programs.append(p)
        outs.append(p.tensor(out, n, H, P))
        first += n
    return _State(programs, outs)


def _exact_ssm(case, r):
    T, H, G, N, P = (case[k] for k in ("tokens", "heads", "groups", "state", "head_dim"))
    xbc, dt, a_log, bias, skip = (t.double() for t in _inputs_ssm(case, r))
    x = xbc[:, :H * P].view(T + 1, H, P)
    B, C = (xbc[:, H * P + i * G * N:H * P + (i + 1) * G * N].view(T + 1, G, N).repeat_interleave(H // G, 1) for i in (0, 1))
    step = torch.nn.functional.softplus(dt + bias)
    decay = torch.exp(-a_log.exp() * step)
    S, out = torch.zeros(H, N, P, dtype=torch.float64, device="cuda"), torch.empty(T + 1, H, P, dtype=torch.float64, device="cuda")
    for t in range(T + 1):
        S = decay[t][:, None, None] * S + (step[t][:, None] * B[t])[:, :, None] * x[t][:, None, :]
        out[t] = torch.einsum("hnp,hn->hp", S, C[t]) + skip[:, None] * x[t]
    return [out[:T], out[T:]]


def _work_ssm(case):
    T, H, G, N, P = (case[k] for k in ("tokens", "heads", "groups", "state", "head_dim"))
    return {"bytes": 4 * ((T + 1) * (2 * H * P + 2 * G * N + H) + 4 * H * N * P), "flops": 5 * (T + 1) * H * N * P}


# ── routed experts ───────────────────────────────────────────────────────────────────────────────────────────────────
def _inputs_moe(case, r):
    T, D, F, E = case["tokens"], case["width"], case["ff"], case["experts"]
    gate, up, down = (r.weight(E * F, D, case["dtype"]), r.weight(E * F, D, case["dtype"]), r.weight(E * D, F, case["dtype"]))
    return gate, up, down, r.normal(T, D), r.normal(T, E)


def _prepare_moe(case, r):
    T, D, F, E, top, wdt = case["tokens"], case["width"], case["ff"], case["experts"], case["top"], WDT[case["dtype"]]
    gate, up, down, x, logits = _inputs_moe(case, r)
    p = _Program()
    src, log, route, out = p.buf(T * D), p.buf(T * E), p.buf(T * top * 2), p.buf(T * D)
    w, o = p.dense(gate, up, down, torch.zeros(E, dtype=gate.dtype, device="cuda"))
    wb = p.ext(w)
    p.ops.append(DeviceOp.route(route, log, wb, o[3], T, E, top, wdt))
    op = DeviceOp.moe_ffn(out, src, route, wb, 0, o[0], o[1], o[2], T, D, F, E, top, wdt, float("inf"), 1.0, up_offset=0.0)
    op.u.seq.buf[4] = p.buf(seq_scratch_elems(op))
    p.ops.append(op)
    p.compile()
    p.tensor(src, T, D).copy_(x)
    p.tensor(log, T, E).copy_(logits)
    return _State([p], p.tensor(out, T, D))


def _exact_moe(case, r):
    T, D, F, E, top = case["tokens"], case["width"], case["ff"], case["experts"], case["top"]
    gate, up, down, x, logits = _inputs_moe(case, r)
    x, share = x.double(), logits.double().softmax(-1)
    out, best = torch.zeros_like(x), share.topk(top, -1).indices
    for e in range(E):
        rows = (best == e).any(-1).nonzero().reshape(-1)
        h = x[rows]
        u = torch.nn.functional.silu(h @ gate[e * F:(e + 1) * F].double().T) * (h @ up[e * F:(e + 1) * F].double().T)
        out[rows] += share[rows, e, None] * (u @ down[e * D:(e + 1) * D].double().T)
    return out


def _work_moe(case):
    T, D, F, E, top = case["tokens"], case["width"], case["ff"], case["experts"], case["top"]
    return {"bytes": min(E, T * top) * 3 * D * F * 2 + 8 * T * D, "flops": 6 * T * top * D * F}
