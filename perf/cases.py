"""The work that a program built on this framework has it do, as cases that can be timed and compared.

A case is one pass of a caller through the public entry points of `muser_b200.operator` on resident weights:

  decode    one decoder layer at decode, GGUF K-quant weights in the Q4_K_M mix (Q6_K for v and down, Q4_K elsewhere):
            input norm + q | k | v | gate in one launch, per-head norms, sigmoid gate, o_proj, sandwich norm, fused
            SwiGLU, down_proj, sandwich norm; f32 activations, 1 to 16 tokens.  Attention is not on this path: the
            normalised q stands in for its output.  With "graph" the step is a CUDA graph made once, as a serving loop
            keeps it; without, every call is issued anew.
  verify    a speculative-verify batch: the layer's seven K-quant projections on activations of several draft tokens
            (2 to 64, bf16 or f32).
  lm_head   the vocabulary projection with scale, soft cap and fused greedy pick (1 to 16 tokens, any K-quant).
  nvfp4     one decoder layer in NVFP4 with on-the-fly NVFP4 activations (W4A4): norm + quantize, q | k | v in one
            launch, o_proj + residual, norm + quantize, SwiGLU that leaves quantized, down_proj + residual; a prompt of
            1 to 32768 tokens.
  nvfp4_a16 the seven projections of a layer whose NVFP4 checkpoint carries no activation scales (weight-only lane).

The large geometry is the framework's benchmark layer (hidden 5120, 40 query and 8 key/value heads of 128, FFN 27648;
202048-row vocabulary); the small one is a 1024-wide layer as the tests use.  Weights and activations are normal with
the deviations a trained layer shows (0.02 and about 1).
"""
from __future__ import annotations

import torch

from muser_b200 import operator as op
from muser_b200 import synth, workloads

HEAD_DIM = 128
EPS, EPS_POST = 1e-5, 1e-8
QUANTS = {"q4_k": synth.Q4_K, "q5_k": synth.Q5_K, "q6_k": synth.Q6_K}
DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}
LARGE = {"hidden": 5120, "heads": 40, "kv_heads": 8, "ffn": 27648}
SMALL = {"hidden": 1024, "heads": 8, "kv_heads": 2, "ffn": 2048}


def listed():
    return [
        # the smallest call: one token through a small layer, issued call by call; launches and their latency count
        dict(name="decode_small_1", kind="decode", **SMALL, tokens=1, graph=False),
        # one sequence decoding through a layer of the large model: the framework's headline (weights from HBM)
        dict(name="decode_1", kind="decode", **LARGE, tokens=1, graph=True),
        # eight sequences decoding together
        dict(name="decode_8", kind="decode", **LARGE, tokens=8, graph=True),
        # speculative verification: a short and a long draft in bf16, and a ragged one in f32
        dict(name="verify_16", kind="verify", **LARGE, tokens=16, dtype="bf16"),
        dict(name="verify_27_f32", kind="verify", **LARGE, tokens=27, dtype="f32"),
        dict(name="verify_64", kind="verify", **LARGE, tokens=64, dtype="bf16"),
        # the greedy next token from the large model's vocabulary
        dict(name="lm_head_1", kind="lm_head", hidden=5120, vocab=202048, quant="q5_k", tokens=1),
        # a checkpoint without activation scales, decoding two sequences
        dict(name="a16_2", kind="nvfp4_a16", **LARGE, tokens=2),
        # NVFP4 at a verify-sized batch, a ragged short prompt, the benchmark's prompt, a long document
        dict(name="nvfp4_16", kind="nvfp4", **LARGE, tokens=16),
        dict(name="nvfp4_509", kind="nvfp4", **LARGE, tokens=509),
        dict(name="nvfp4_2048", kind="nvfp4", **LARGE, tokens=2048),
        dict(name="nvfp4_32768", kind="nvfp4", **LARGE, tokens=32768),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(lo * (hi / lo) ** rng.random())))


def _geometry(rng, step):
    """A layer between the small and the large one; every width a multiple of `step`."""
    hidden = step * rng.randint(-(-1024 // step), 5120 // step)
    heads = 2 * rng.randint(4, 20)
    kv_heads = rng.choice([h for h in (1, 2, 4, 5, 8, 10, 20) if heads % h == 0])
    ffn = min(27648, step * round(hidden * rng.uniform(2.0, 5.4) / step))
    return {"hidden": hidden, "heads": heads, "kv_heads": kv_heads, "ffn": ffn}


def draw(rng):
    kind = rng.choice(["decode", "decode", "verify", "verify", "lm_head", "nvfp4_a16", "nvfp4", "nvfp4", "nvfp4"])
    if kind == "decode":
        return dict(kind=kind, **_geometry(rng, 256), tokens=rng.randint(1, 16), graph=rng.random() < 0.7)
    if kind == "verify":
        return dict(kind=kind, **_geometry(rng, 256), tokens=_log_int(rng, 2, 64), dtype=rng.choice(["bf16", "bf16", "f32"]))
    if kind == "lm_head":
        return dict(kind=kind, hidden=256 * rng.randint(4, 20), vocab=_log_int(rng, 32000, 202048), quant=rng.choice(sorted(QUANTS)),
                    tokens=rng.randint(1, 16))
    if kind == "nvfp4_a16":
        return dict(kind=kind, **_geometry(rng, 256), tokens=rng.randint(1, 16))
    return dict(kind=kind, **_geometry(rng, 64), tokens=_log_int(rng, 1, 32768))


# ---------------------------------------------------------------------------------------------------- geometry


def _projections(case):
    """name -> (n_in, n_out, K-quant dtype of the Q4_K_M mix)."""
    h, a, kv, f = case["hidden"], case["heads"] * HEAD_DIM, case["kv_heads"] * HEAD_DIM, case["ffn"]
    p = {"q": (h, a, synth.Q4_K), "k": (h, kv, synth.Q4_K), "v": (h, kv, synth.Q6_K), "o": (a, h, synth.Q4_K),
         "ffn_gate": (h, f, synth.Q4_K), "ffn_up": (h, f, synth.Q4_K), "ffn_down": (f, h, synth.Q6_K)}
    if case["kind"] == "decode":
        p["gate"] = (h, a, synth.Q4_K)
    return p


def work(case):
    t = case["tokens"]
    if case["kind"] == "lm_head":
        k, n = case["hidden"], case["vocab"]
        return {"bytes": n * (k // 256) * synth.BLOCK_BYTES[QUANTS[case["quant"]]] + t * k * 2 + t * n * 4 + t * 12, "flops": 2 * t * n * k}
    p = _projections(case)
    macs = sum(k * n for k, n, _ in p.values())
    h, a, kv, f = case["hidden"], case["heads"] * HEAD_DIM, case["kv_heads"] * HEAD_DIM, case["ffn"]
    if case["kind"] in ("decode", "verify"):
        weights = sum(n * (k // 256) * synth.BLOCK_BYTES[dt] for k, n, dt in p.values())
    else:
        weights = macs // 2 + macs // 16  # codes and one scale per 16
    if case["kind"] == "decode":  # hidden in and out, q, k, v, gate, the two normed rows and the FFN activation out
        acts = t * 4 * (4 * h + 2 * a + 2 * kv + f)
    elif case["kind"] == "nvfp4":
        acts = t * 2 * (3 * h + a + 2 * kv)
    else:
        x = DTYPES[case.get("dtype", "bf16")].itemsize
        acts = t * (x * (2 * h + a + f) + (2 if case["kind"] == "nvfp4_a16" else 4) * (a + 2 * kv + 2 * h + 2 * f))
    return {"bytes": weights + acts, "flops": 2 * t * macs}


def tolerance(case):
    if case["kind"] == "nvfp4_a16":
        return "exact"  # an integer lane with a fixed order of the four roundings behind it
    # about four times what the path shows against itself in 64 bits on the large geometry
    if case["kind"] == "nvfp4":  # bf16 outputs; a last-bit difference can move the next projection's input to another 4-bit code
        return {"rel": 6.5e-3, "max": 0.5}
    if case["kind"] == "decode":  # 15-bit activations through four projections in a row
        return {"rel": 7e-4, "max": 4e-3}
    if case["kind"] == "verify":
        return {"rel": 4.3e-4, "max": 2e-3}
    return {"rel": 2.2e-4, "max": 1e-3, "differ": 0.0}


# ---------------------------------------------------------------------------------------------------- state


def _decode_inputs(case, seed):
    """Norm weights, the per-head ones of q and k, and the hidden state."""
    g = torch.Generator("cuda").manual_seed((seed << 8) + 1)
    rand = lambda *s: torch.randn(s, device="cuda", generator=g)  # noqa: E731
    norms = {n: 1.0 + 0.1 * rand(case["hidden"]) for n in ("attn", "post_attn", "ffn", "post_ffn")}
    q_norm, k_norm = 0.0884 + 0.01 * rand(HEAD_DIM), 1.0 + 0.1 * rand(HEAD_DIM)
    return norms, q_norm, k_norm, rand(case["tokens"], case["hidden"])


class _Decode:
    def __init__(self, case, seed):
        t, p = case["tokens"], _projections(case)
        self.case, self.t = case, t
        self.ctx = op.Context(0, workspace_bytes=1 << 20)
        self.kern = op.CudaKernels(self.ctx)
        self.w = _kquant_weights(self.ctx, p, seed)
        self.norms, self.q_norm, self.k_norm, self.embedding = _decode_inputs(case, seed)
        new = lambda n: torch.empty((t, n), device="cuda")  # noqa: E731
        self.hidden, self.y, self.proj, self.down = (new(case["hidden"]) for _ in range(4))
        self.out = {n: new(p[n][1]) for n in ("q", "k", "v", "gate")}
        self.act = new(case["ffn"])
        self.step = workloads.capture(self.layer) if case["graph"] else self.layer

    def layer(self):
        k, w, t, n, o = self.kern, self.w, self.t, self.norms, self.out
        self.hidden.copy_(self.embedding)
        norm = {"norm_weight": n["attn"], "norm_eps": EPS}
        k.encode_quantized_matmul_group([w["q"], w["k"], w["v"], w["gate"]], self.hidden, [o["q"], o["k"], o["v"], o["gate"]], t,
                                        epilogues=[norm] * 4)
        k.encode_head_rms_norm(o["q"], self.q_norm, EPS, self.case["heads"])
        k.encode_head_rms_norm(o["k"], self.k_norm, EPS, self.case["kv_heads"])
        k.encode_sigmoid_gate(o["q"], o["gate"])
        k.encode_quantized_matmul(w["o"], o["q"], self.proj, t)
        k.encode_fused_norm_residual_rms_norm(self.hidden, self.proj, n["post_attn"], EPS_POST, self.y, n["ffn"], EPS)
        k.encode_ffn_gate_up_silu(w["ffn_gate"], w["ffn_up"], self.y, self.act, t)
        k.encode_quantized_matmul(w["ffn_down"], self.act, self.down, t)
        k.encode_fused_norm_residual_rms_norm(self.hidden, self.down, n["post_ffn"], EPS_POST)

    def run(self):
        self.step()
        return {"hidden": self.hidden, "y": self.y, "proj": self.proj, "act": self.act, "down": self.down, **self.out}


INPUT = {"q": "attn", "k": "attn", "v": "attn", "o": "o", "ffn_gate": "ffn", "ffn_up": "ffn", "ffn_down": "down"}


def _projection_inputs(case, seed):
    p, g = _projections(case), torch.Generator("cuda").manual_seed((seed << 8) + 1)
    return {i: torch.randn((case["tokens"], p[n][0]), device="cuda", generator=g).to(DTYPES[case.get("dtype", "bf16")]) for n, i in INPUT.items()}


class _Projections:
    """The seven projections of a layer, each on its own input (q, k and v share one, gate and up another)."""

    def __init__(self, case, seed):
        t, p = case["tokens"], _projections(case)
        self.t = t
        a16 = case["kind"] == "nvfp4_a16"
        self.ctx = op.Context(0, workspace_bytes=(2 * t * max(k for k, _, _ in p.values()) if a16 else 0) + (1 << 20))
        self.kern = op.CudaKernels(self.ctx)
        self.w = _nvfp4_weights(self.ctx, p, seed, {})[0] if a16 else _kquant_weights(self.ctx, p, seed)
        self.encode = self.kern.encode_nvfp4_matmul if a16 else self.kern.encode_quantized_matmul
        self.x = _projection_inputs(case, seed)
        self.y = {n: torch.empty((t, p[n][1]), device="cuda", dtype=torch.float16 if a16 else torch.float32) for n in p}

    def run(self):
        for n, y in self.y.items():
            self.encode(self.w[n], self.x[INPUT[n]], y, self.t)
        return self.y


def _lm_head_inputs(case, seed):
    k, n, dt = case["hidden"], case["vocab"], QUANTS[case["quant"]]
    rows = -(-n // 8)
    raw = torch.cat([synth.quantize_kquant(synth.normal_weights(min(rows, n - r), k, seed=seed, stream=90 + r, device="cuda"), dt) for r in range(0, n, rows)])
    return raw, synth.normal_activations(case["tokens"], k, seed=seed, device="cuda")


class _LmHead:
    def __init__(self, case, seed):
        k, n, dt = case["hidden"], case["vocab"], QUANTS[case["quant"]]
        self.t = case["tokens"]
        self.ctx = op.Context(0, workspace_bytes=1 << 20)
        self.kern = op.CudaKernels(self.ctx)
        raw, self.x = _lm_head_inputs(case, seed)
        self.w = op.Weight(self.ctx, op.TensorView(raw, dt, k, n))
        self.logits = torch.empty((self.t, n), device="cuda")

    def run(self):
        picked = self.kern.encode_lm_head_argmax(self.w, self.x, self.t, logits=self.logits, out_scale=0.5, softcap=30.0)
        return [*picked, self.logits]


def _nvfp4_inputs(case, seed):
    """The hidden state, the two norms' weights and rows to calibrate with."""
    h, g = case["hidden"], torch.Generator("cuda").manual_seed((seed << 8) + 1)
    x = torch.randn((case["tokens"], h), device="cuda", generator=g).to(torch.bfloat16)
    norms = [1.0 + 0.1 * torch.randn(h, device="cuda", generator=g) for _ in range(2)]
    return x, norms, torch.randn((128, h), device="cuda", generator=g)


class _Nvfp4Layer:
    def __init__(self, case, seed):
        t, p, h = case["tokens"], _projections(case), case["hidden"]
        a = p["q"][1]
        self.t = t
        self.ctx = op.Context(0, workspace_bytes=(t + 128) * (a // 2 + a // 16) + (1 << 20))
        self.kern = op.CudaKernels(self.ctx)
        self.x, self.norms, sample = _nvfp4_inputs(case, seed)
        self.w, self.isi = _nvfp4_weights(self.ctx, p, seed, {"sample": sample, "norms": self.norms})
        new = lambda n: torch.empty((t, n), device="cuda", dtype=torch.bfloat16)  # noqa: E731
        self.q, self.k, self.v, self.h1, self.h2 = new(a), new(p["k"][1]), new(p["v"][1]), new(h), new(h)
        quantized = lambda n: (torch.empty((t, n // 2), dtype=torch.uint8, device="cuda"),  # noqa: E731
                               torch.empty(-(-t // 128) * (n // 64) * 512, dtype=torch.uint8, device="cuda"))
        self.xq, self.fq = quantized(h), quantized(case["ffn"])

    def run(self):
        k, w, t = self.kern, self.w, self.t
        k.quantize_nvfp4_activation(self.x, self.isi["q"], norm_weight=self.norms[0], norm_eps=EPS, out=self.xq)
        k.encode_nvfp4_group_prequant([w["q"], w["k"], w["v"]], *self.xq, [self.q, self.k, self.v], t)
        k.encode_nvfp4_matmul(w["o"], self.q, self.h1, t, residual=self.x)
        k.quantize_nvfp4_activation(self.h1, self.isi["ffn_gate"], norm_weight=self.norms[1], norm_eps=EPS, out=self.xq)
        k.encode_nvfp4_ffn_gate_up_silu_requant(w["ffn_gate"], w["ffn_up"], *self.xq, t, self.isi["ffn_down"], out_packed=self.fq[0], out_scales=self.fq[1])
        k.encode_nvfp4_prequant(w["ffn_down"], *self.fq, self.h2, t, residual=self.h1)
        return [self.q, self.k, self.v, self.h1, self.h2]


def _kquant_raw(p, seed):
    """name -> K-quant blocks of the projection's weights."""
    return {name: synth.quantize_kquant(synth.normal_weights(n, k, seed=seed, stream=i, device="cuda"), dt) for i, (name, (k, n, dt)) in enumerate(p.items())}


def _kquant_weights(ctx, p, seed):
    return {name: op.Weight(ctx, op.TensorView(raw, p[name][2], p[name][0], p[name][1])) for name, raw in _kquant_raw(p, seed).items()}


def _nvfp4_raw(p, seed, calibration):
    """name -> (codes, scales, scale2) and, given calibration rows, each projection's input_scale_inv as a checkpoint
    stores it (from the largest magnitude that the sample shows at that input, with a margin); without them the
    weight-only form."""
    dense = {n: synth.normal_weights(o, i, seed=seed, stream=s, device="cuda") for s, (n, (i, o, _)) in enumerate(p.items())}
    isi = dict.fromkeys(p)
    if calibration:
        x = calibration["sample"]
        normed = [x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * w for w in calibration["norms"]]
        ffn = torch.nn.functional.silu(normed[1] @ dense["ffn_gate"].t()) * (normed[1] @ dense["ffn_up"].t())
        inputs = {"q": normed[0], "o": normed[0] @ dense["q"].t(), "ffn_gate": normed[1], "ffn_down": ffn}
        isi.update({n: synth.activation_input_scale_inv(1.25 * v) for n, v in inputs.items()})
        isi["k"] = isi["v"] = isi["q"]
        isi["ffn_up"] = isi["ffn_gate"]
    return {n: synth.nvfp4_weight(dense.pop(n)) for n in p}, isi


def _nvfp4_weights(ctx, p, seed, calibration):
    raw, isi = _nvfp4_raw(p, seed, calibration)
    return {n: op.Weight(ctx, op.TensorView(packed, op.NVFP4, p[n][0], p[n][1], scales, scale2, isi[n])) for n, (packed, scales, scale2) in raw.items()}, isi


def prepare(case, seed):
    return {"decode": _Decode, "verify": _Projections, "lm_head": _LmHead, "nvfp4_a16": _Projections, "nvfp4": _Nvfp4Layer}[case["kind"]](case, seed)


def run(state):
    return state.run()


# ---------------------------------------------------------------------------------------------------- in 64 bits


def _f16_pairs(b):
    return b.contiguous().view(torch.float16).double()


def _dense64(raw, dt):
    """[rows][blocks * bytes] K-quant blocks -> f64 weights."""
    b = raw.reshape(raw.shape[0], -1, synth.BLOCK_BYTES[dt])
    if dt == synth.Q6_K:
        ql, qh = b[..., :128].reshape(*b.shape[:2], 2, 2, 32), b[..., 128:192].reshape(*b.shape[:2], 2, 32)
        lo = torch.stack([ql[..., 0, :] & 15, ql[..., 1, :] & 15, ql[..., 0, :] >> 4, ql[..., 1, :] >> 4], -2)
        hi = torch.stack([(qh >> s) & 3 for s in (0, 2, 4, 6)], -2)
        q = (lo | (hi << 4)).reshape(*b.shape[:2], 16, 16).double() - 32.0
        sc = b[..., 192:208].contiguous().view(torch.int8).double()
        return (q * (sc * _f16_pairs(b[..., 208:210])).unsqueeze(-1)).reshape(b.shape[0], -1)
    packed = b[..., 4:16]
    low, mid, top = packed[..., 0:4], packed[..., 4:8], packed[..., 8:12]
    sc = torch.cat([low & 63, (top & 15) | ((low >> 6) << 4)], -1).double() * _f16_pairs(b[..., 0:2])
    mn = torch.cat([mid & 63, (top >> 4) | ((mid >> 6) << 4)], -1).double() * _f16_pairs(b[..., 2:4])
    qs = b[..., -128:].reshape(*b.shape[:2], 4, 32)
    q = torch.stack([qs & 15, qs >> 4], -2).reshape(*b.shape[:2], 8, 32)
    if dt == synth.Q5_K:
        q = q | torch.stack([((b[..., 16:48] >> j) & 1) << 4 for j in range(8)], -2)
    return (q.double() * sc.unsqueeze(-1) - mn.unsqueeze(-1)).reshape(b.shape[0], -1)


def _product64(x, rows, decode):
    """x [tokens][n_in] times the weights' transpose, decoded some rows at a time."""
    step = max(1, (1 << 26) // x.shape[1])
    return torch.cat([x.double() @ decode(r, min(rows, r + step)).t() for r in range(0, rows, step)], 1)


def _kquant64(raw, dt, x):
    return _product64(x, raw.shape[0], lambda a, b: _dense64(raw[a:b], dt))


def _norm64(x, w, eps):
    x = x.double()
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w.double()


_E2M1 = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0, -0.0, -0.5, -1.0, -1.5, -2.0, -3.0, -4.0, -6.0)


def _fp4_values(packed, scales):
    """Codes and their E4M3 scales, one per 16 -> f64 values."""
    codes = torch.stack([packed & 15, packed >> 4], -1).reshape(packed.shape[0], -1, 16)
    return (torch.tensor(_E2M1, dtype=torch.float64, device=packed.device)[codes.int()] * scales.view(torch.float8_e4m3fn).double().unsqueeze(-1)).flatten(1)


def _nvfp4_dot64(w, x):
    """x (codes times scales, or any f64 values) times an NVFP4 weight."""
    packed, scales, scale2 = w
    return _product64(x, packed.shape[0], lambda a, b: _fp4_values(packed[a:b], scales[a:b])) * scale2


def _fp4_round(x, isi):
    """x as the W4A4 lane's inputs: each 16 values of f16(x) * isi as E2M1 codes times an E4M3 scale, over isi."""
    r = x.half().float().reshape(x.shape[0], -1, 16)
    isi = torch.tensor(isi, dtype=torch.float32, device=x.device)
    scale = (r.abs().amax(-1) * torch.tensor(1.0 / 6.0, dtype=torch.float32, device=x.device) * isi).clamp_max(448.0).to(torch.float8_e4m3fn).float().unsqueeze(-1)
    mag, code = r.abs() * isi, 0
    for edge, inclusive in ((0.25, False), (0.75, True), (1.25, False), (1.75, True), (2.5, False), (3.5, True), (5.0, False)):
        code = code + ((mag >= scale * edge) if inclusive else (mag > scale * edge)).int()
    value = torch.tensor(_E2M1[:8], dtype=torch.float64, device=x.device)[code] * scale
    return torch.copysign(value, r.double()).flatten(1) / isi.double()


def _int8_round(x):
    """x as the weight-only lane's inputs: each 256 values of f16(x) as int8 against the first of largest magnitude."""
    r = x.half().float().reshape(x.shape[0], -1, 256)
    inverse = -127.0 / r.gather(-1, r.abs().argmax(-1, keepdim=True))
    return (torch.round(inverse.double() * r.double()).clamp_max(127.0) * (1.0 / inverse).double()).flatten(1)


def _exact_decode(case, seed):
    p = _projections(case)
    raw = _kquant_raw(p, seed)
    norms, q_norm, k_norm, hidden = _decode_inputs(case, seed)
    dot = lambda n, x: _kquant64(raw[n], p[n][2], x)  # noqa: E731
    heads = lambda x, w: _norm64(x.reshape(case["tokens"], -1, HEAD_DIM), w, EPS).flatten(1)  # noqa: E731
    x = _norm64(hidden, norms["attn"], EPS)
    q, k, v, gate = heads(dot("q", x), q_norm), heads(dot("k", x), k_norm), dot("v", x), dot("gate", x)
    q = q * torch.sigmoid(gate)
    proj = dot("o", q)
    hidden = hidden.double() + _norm64(proj, norms["post_attn"], EPS_POST)
    y = _norm64(hidden, norms["ffn"], EPS)
    act = torch.nn.functional.silu(dot("ffn_gate", y)) * dot("ffn_up", y)
    down = dot("ffn_down", act)
    return {"hidden": hidden + _norm64(down, norms["post_ffn"], EPS_POST), "y": y, "proj": proj, "act": act, "down": down, "q": q, "k": k, "v": v, "gate": gate}


def _exact_projections(case, seed):
    p, x = _projections(case), _projection_inputs(case, seed)
    if case["kind"] == "verify":
        raw = _kquant_raw(p, seed)
        return {n: _kquant64(raw[n], p[n][2], x[INPUT[n]]) for n in p}
    raw = _nvfp4_raw(p, seed, {})[0]
    return {n: _nvfp4_dot64(raw[n], _int8_round(x[INPUT[n]])) for n in p}


def _exact_lm_head(case, seed):
    raw, x = _lm_head_inputs(case, seed)
    logits = 30.0 * torch.tanh(_kquant64(raw, QUANTS[case["quant"]], x) * 0.5 / 30.0)
    return [None, logits.amax(-1), None, logits]


def _exact_nvfp4(case, seed):
    """What one entry point hands to the next has the type that the caller's buffers have: bf16, or 4-bit codes."""
    x, norms, sample = _nvfp4_inputs(case, seed)
    w, isi = _nvfp4_raw(_projections(case), seed, {"sample": sample, "norms": norms})
    stored = lambda v: v.float().bfloat16()  # noqa: E731
    a = _fp4_round(_norm64(x, norms[0], EPS), isi["q"])
    q, k, v = (_nvfp4_dot64(w[n], a) for n in ("q", "k", "v"))
    h1 = _nvfp4_dot64(w["o"], _fp4_round(stored(q), isi["o"])) + x.double()
    a = _fp4_round(_norm64(stored(h1), norms[1], EPS), isi["ffn_gate"])
    act = torch.nn.functional.silu(_nvfp4_dot64(w["ffn_gate"], a).half().double()) * _nvfp4_dot64(w["ffn_up"], a).half().double()
    return [q, k, v, h1, _nvfp4_dot64(w["ffn_down"], _fp4_round(act, isi["ffn_down"])) + stored(h1).double()]


def exact(case, seed):
    """run()'s outputs for prepare(case, seed)'s inputs in plain 64-bit arithmetic, from the formats' definitions."""
    return {"decode": _exact_decode, "verify": _exact_projections, "nvfp4_a16": _exact_projections, "lm_head": _exact_lm_head, "nvfp4": _exact_nvfp4}[case["kind"]](case, seed)
