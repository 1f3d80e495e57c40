"""What is timed: the quantized-linear operators as a serving program calls them.

Five kinds of work, each over the sizes it sees in use:

* ``awq_layer``: the AWQ 4-bit linears of one decoder layer in the order a forward pass calls them (fused
  query/key/value projection, output projection, gated feed-forward projection, down projection), from one
  sequence being decoded to a long prompt.
* ``gptq``: one GPTQ 4-bit linear, symmetric or with zero points.
* ``gguf``: one linear on GGUF blocks, from a single small projection to the vocabulary projection.
* ``fp8``: one E4M3 linear with 128 x 128 block scales.
* ``moe``: the MXFP4 mixture-of-experts feed-forward layer, router included.

Weights are made on the GPU with the distributions of ``oxydllm_b200/synth.py``: uniform 4-bit codes with scales
|N(0, 0.02)| / 7 + 1e-4, N(0, 0.02) weights for FP8 and MXFP4, well-formed GGUF blocks of about that spread.
Activations are bf16 N(0, 1).
"""
import math

import torch

from oxydllm_b200 import formats as F
from oxydllm_b200.linear import Fp8Linear, GatedFfnProjection, PackedQuantLinear, QLinear, QuantWeight
from oxydllm_b200.moe import GptOssMoe

GGUF_TYPES = {"Q4_0": F.GGML_Q4_0, "Q8_0": F.GGML_Q8_0, "Q4_K": F.GGML_Q4_K, "Q6_K": F.GGML_Q6_K}


# ------------------------------------------------------------------------------------------------------- the cases
def _awq_layer(tokens, hidden=4096, kv=1024, inter=14336, group=128):
    return {"kind": "awq_layer", "tokens": tokens, "hidden": hidden, "kv": kv, "inter": inter, "group": group}


def _gptq(tokens, k, n, group=128, sym=False):
    return {"kind": "gptq", "tokens": tokens, "k": k, "n": n, "group": group, "sym": sym}


def _gguf(tokens, k, n, type_):
    return {"kind": "gguf", "tokens": tokens, "k": k, "n": n, "type": type_}


def _fp8(tokens, k, n):
    return {"kind": "fp8", "tokens": tokens, "k": k, "n": n}


def _moe(tokens, experts=32, hidden=2880, inter=2880):
    return {"kind": "moe", "tokens": tokens, "experts": experts, "hidden": hidden, "inter": inter, "top_k": 4}


def listed():
    return [
        # The smallest call: one attention-sized projection of a GGUF model, one sequence being decoded.
        {"name": "gguf_q4k_decode_1", **_gguf(1, 4096, 4096, "Q4_K")},
        # Interactive use of an AWQ model: one sequence, every linear of a layer once.
        {"name": "awq_layer_decode_1", **_awq_layer(1)},
        # A server with a dozen sequences in its decode batch.
        {"name": "awq_layer_decode_12", **_awq_layer(12)},
        # A well filled continuous batch on a smaller model with 64-wide groups; 77 is no multiple of anything.
        {"name": "awq_layer_batch_77", **_awq_layer(77, hidden=3072, inter=8192, group=64)},
        # Prefill of a long prompt.
        {"name": "awq_layer_prefill_2048", **_awq_layer(2048)},
        # GPTQ decode batch on the widest projection.
        {"name": "gptq_decode_6", **_gptq(6, 4096, 14336)},
        # FP8 decode of one sequence, and a medium prompt.
        {"name": "fp8_decode_1", **_fp8(1, 4096, 14336)},
        {"name": "fp8_prefill_600", **_fp8(600, 4096, 14336)},
        # Vocabulary projection of a GGUF model (these are usually kept in Q6_K) for three sequences.
        {"name": "gguf_q6k_vocab_3", **_gguf(3, 4096, 128256, "Q6_K")},
        # Mixture-of-experts layer: two sequences, a continuous batch, and a long prompt.
        {"name": "moe_decode_2", **_moe(2)},
        {"name": "moe_batch_50", **_moe(50)},
        {"name": "moe_prefill_4096", **_moe(4096)},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["awq_layer", "awq_layer", "gptq", "gguf", "fp8", "moe"])
    if kind == "awq_layer":
        return _awq_layer(_log_int(rng, 1, 2048), hidden=rng.choice([2048, 2560, 3072, 4096]), kv=rng.choice([512, 1024]),
                          inter=rng.choice([5632, 8192, 9728, 11008, 14336]), group=rng.choice([128, 128, 64, 32]))
    if kind == "gptq":
        return _gptq(_log_int(rng, 1, 512), rng.choice([2048, 3072, 4096, 14336]), rng.choice([1024, 4096, 6144, 14336]),
                     rng.choice([128, 128, 64]), rng.random() < 0.5)
    if kind == "gguf":
        type_ = rng.choice(sorted(GGUF_TYPES))
        if rng.random() < 0.25:  # vocabulary projection of a few sequences
            return _gguf(_log_int(rng, 1, 8), rng.choice([2048, 4096]), 8 * _log_int(rng, 4000, 16032), type_)
        return _gguf(_log_int(rng, 1, 512), rng.choice([2048, 4096, 14336]), rng.choice([1024, 4096, 6144, 14336]), type_)
    if kind == "fp8":
        return _fp8(_log_int(rng, 1, 2048), rng.choice([2048, 4096, 7168]), rng.choice([1024, 4096, 6144, 14336]))
    return _moe(_log_int(rng, 1, 4096), experts=rng.choice([16, 32]), hidden=rng.choice([2048, 2880]),
                inter=rng.choice([1024, 2048, 2880]))


# ------------------------------------------------------------------------------------------------- inputs and weights
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _x(g, m, k):
    return torch.randn(m, k, generator=g, device="cuda", dtype=torch.float32).to(torch.bfloat16)


def _words(g, *shape):
    return torch.randint(-2**31, 2**31, shape, generator=g, device="cuda", dtype=torch.int64).to(torch.int32)


def _bytes(g, *shape):
    return torch.randint(0, 256, shape, generator=g, device="cuda", dtype=torch.uint8)


def _scales(g, groups, n):
    return (torch.randn(groups, n, generator=g, device="cuda").abs() * 0.02 / 7.0 + 1e-4).to(torch.float16)


def _awq(g, k, n, group):
    return _words(g, k, n // 8), _words(g, k // group, n // 8), _scales(g, k // group, n)


def _f16_bytes(v):
    return v.to(torch.float16).contiguous().view(torch.uint8).reshape(*v.shape, 2)


def _gguf_blocks(g, type_, n, k):
    """Raw blocks ``[n, blocks, bytes]``: random codes, block scales that give weights of about N(0, 0.02)'s spread."""
    per, _ = F.GGML_BLOCK[GGUF_TYPES[type_]]
    nb = k // per
    spread = torch.rand(n, nb, generator=g, device="cuda") * 0.5 + 0.75
    if type_ == "Q4_0":  # d (q - 8)
        parts = [_f16_bytes(spread * 0.004), _bytes(g, n, nb, 16)]
    elif type_ == "Q8_0":  # d q
        parts = [_f16_bytes(spread * 0.0003), _bytes(g, n, nb, 32)]
    elif type_ == "Q4_K":  # (d sc) q - dmin mn: 6-bit sc and mn
        parts = [_f16_bytes(spread * 1.2e-4), _f16_bytes(spread * 9e-4), _bytes(g, n, nb, 12), _bytes(g, n, nb, 128)]
    else:  # Q6_K: (d sc) (q - 32), 8-bit signed sc; quants first, d last
        parts = [_bytes(g, n, nb, 192), _bytes(g, n, nb, 16), _f16_bytes(spread * 1.5e-5)]
    return torch.cat(parts, dim=-1).reshape(-1)


def _mxfp4(g, rows, k):
    """N(0, 0.02) weights as E2M1 codes with one E8M0 scale per 32 (blocks ``[rows, k/32, 16]``, low nibble first)."""
    w = torch.randn(rows, k // 32, 32, generator=g, device="cuda") * 0.02
    e = torch.floor(torch.log2(w.abs().amax(-1).clamp_min(1e-30))) - 2
    mag = (w / torch.exp2(e)[..., None]).abs()
    mid = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0], device="cuda")
    code = torch.bucketize(mag, mid).to(torch.uint8) | ((w < 0).to(torch.uint8) << 3)
    return (code[..., 0::2] | (code[..., 1::2] << 4)).contiguous(), (e + 127).to(torch.uint8)


def _mxfp4_experts(g, experts, rows, k):
    made = [_mxfp4(g, rows, k) for _ in range(experts)]
    return torch.stack([b for b, _ in made]), torch.stack([s for _, s in made])


def _inputs(case, seed):
    """The tensors of a case: activations and packed weights as a checkpoint holds them."""
    g = _gen(seed)
    m, kind = case["tokens"], case["kind"]
    if kind == "awq_layer":
        h, i, grp = case["hidden"], case["inter"], case["group"]
        return {"x": _x(g, m, h), "attn": _x(g, m, h), "ffn_in": _x(g, m, h), "qkv": _awq(g, h, h + 2 * case["kv"], grp),
                "o": _awq(g, h, h, grp), "ffn": _awq(g, h, 2 * i, grp), "down": _awq(g, i, h, grp)}
    if kind == "moe":
        e, h, i = case["experts"], case["hidden"], case["inter"]
        gate_up, down = _mxfp4_experts(g, e, 2 * i, h), _mxfp4_experts(g, e, h, i)
        small = lambda *shape: (torch.randn(*shape, generator=g, device="cuda") * 0.02).to(torch.bfloat16)  # noqa: E731
        return {"gate_up": gate_up, "gate_up_bias": small(e, 2 * i), "down": down, "down_bias": small(e, h),
                "router": small(e, h), "router_bias": small(e), "x": _x(g, m, h)}
    k, n = case["k"], case["n"]
    if kind == "gptq":
        zeros = None if case["sym"] else _words(g, k // case["group"], n // 8)
        weight = _words(g, k // 8, n), zeros, _scales(g, k // case["group"], n)
    elif kind == "gguf":
        weight = _gguf_blocks(g, case["type"], n, k)
    else:
        w = torch.randn(n // 128, 128, k // 128, 128, generator=g, device="cuda") * 0.02
        scale = w.abs().amax(dim=(1, 3)) / 448.0
        weight = (w / scale[:, None, :, None]).clamp(-448.0, 448.0).reshape(n, k).to(torch.float8_e4m3fn), scale
    return {"x": _x(g, m, k), "weight": weight}


def prepare(case, seed):
    t, kind = _inputs(case, seed), case["kind"]
    if kind == "awq_layer":
        lin = {name: PackedQuantLinear(QuantWeight.new_awq(4, *t[name])) for name in ("qkv", "o", "ffn", "down")}
        return {"kind": kind, "x": t["x"], "attn": t["attn"], "ffn_in": t["ffn_in"], "qkv": lin["qkv"], "o": lin["o"],
                "ffn": GatedFfnProjection(lin["ffn"], "silu"), "down": lin["down"]}
    if kind == "moe":
        layer = GptOssMoe(*t["gate_up"], t["gate_up_bias"], *t["down"], t["down_bias"], case["hidden"], case["inter"],
                          top_k=case["top_k"], router_weight=t["router"], router_bias=t["router_bias"])
    elif kind == "gptq":
        layer = PackedQuantLinear(QuantWeight.new_gptq(4, case["sym"], *t["weight"]))
    elif kind == "gguf":
        layer = QLinear(GGUF_TYPES[case["type"]], t["weight"], case["n"], case["k"])
    else:
        layer = Fp8Linear(*t["weight"])
    return {"kind": kind, "x": t["x"], "layer": layer}


def run(state):
    if state["kind"] != "awq_layer":
        return state["layer"].forward(state["x"])
    act = state["ffn"].forward(state["ffn_in"])
    return {"qkv": state["qkv"].forward(state["x"]), "o": state["o"].forward(state["attn"]), "ffn": act,
            "down": state["down"].forward(act)}


# --------------------------------------------------------------------------------------------------------- yardsticks
def _int4_bytes(k, n, group, zeros=True):
    return k * n / 2 + (k // group) * (n / 2 if zeros else 0) + (k // group) * n * 2


def work(case):
    m, kind = case["tokens"], case["kind"]
    if kind == "awq_layer":
        h, i, grp = case["hidden"], case["inter"], case["group"]
        q = h + 2 * case["kv"]
        weights = sum(_int4_bytes(k, n, grp) for k, n in ((h, q), (h, h), (h, 2 * i), (i, h)))
        # activations: three inputs, four outputs, and the gated product read again by the down projection
        return {"bytes": weights + 2 * m * (3 * h + q + h + 2 * i + h), "flops": 2 * m * (h * q + h * h + 3 * h * i)}
    if kind == "moe":
        e, h, i, top = case["experts"], case["hidden"], case["inter"], case["top_k"]
        hit = e * (1.0 - (1.0 - top / e) ** m)  # experts that some token is expected to choose
        per_expert = 3 * h * i * 17 / 32 + 2 * (2 * i + h)
        return {"bytes": hit * per_expert + 2 * (e * h + e) + 2 * m * 2 * h, "flops": 2 * m * (top * 3 * h * i + e * h)}
    k, n = case["k"], case["n"]
    if kind == "gptq":
        weights = _int4_bytes(k, n, case["group"], not case["sym"])
    elif kind == "gguf":
        per, size = F.GGML_BLOCK[GGUF_TYPES[case["type"]]]
        weights = n * (k // per) * size
    else:
        weights = n * k + (n // 128) * (k // 128) * 4
    return {"bytes": weights + 2 * m * (k + n), "flops": 2 * m * k * n}


def tolerance(case):
    """About four times the error against the same operation in 64 bits with exact weights.

    One linear is off by 1.7e-3 (bf16 results) to 2.4e-3 (bf16 weights too), largest single value 1.2e-2; the AWQ
    layer by up to 4.5e-3 at its down projection and 3.8e-2 in one gated value (the decode path keeps gate and up in
    bf16 before it multiplies them); the expert layer by 3.0e-3 and 1.9e-2.
    """
    return {"awq_layer": {"rel": 1.8e-2, "max": 0.15}, "moe": {"rel": 1.2e-2, "max": 0.075}}.get(
        case["kind"], {"rel": 1e-2, "max": 0.05})


# ---------------------------------------------------------------------------------------- the same in 64 bits, plain torch
def _nibbles(words, order):
    """The eight 4-bit codes of each 32-bit word, as a last dimension: code ``c`` from nibble ``order[c]``."""
    return torch.stack([(words >> (4 * s)) & 15 for s in order], dim=-1)


def _awq64(qweight, qzeros, scales):
    k, (groups, n) = qweight.shape[0], scales.shape
    order = (0, 4, 1, 5, 2, 6, 3, 7)  # the nibble that holds column 0, 1, ... of a word
    q = _nibbles(qweight, order).reshape(groups, k // groups, n)
    z = _nibbles(qzeros, order).reshape(groups, 1, n)
    return ((q - z) * scales.double()[:, None]).reshape(k, n)


def _gptq64(qweight, qzeros, scales):
    (rows, n), groups = qweight.shape, scales.shape[0]
    q = _nibbles(qweight, range(8)).permute(0, 2, 1).reshape(groups, 8 * rows // groups, n)
    z = 8 if qzeros is None else _nibbles(qzeros, range(8)).reshape(groups, 1, n) + 1
    return ((q - z) * scales.double()[:, None]).reshape(8 * rows, n)


def _f16(raw):
    return raw.contiguous().view(torch.float16).double()


def _gguf64(type_, raw, n, k):
    """``[n, k]`` from raw blocks."""
    per, size = F.GGML_BLOCK[GGUF_TYPES[type_]]
    b = raw.reshape(n, k // per, size)
    if type_ == "Q4_0":
        q = torch.cat([b[..., 2:] & 15, b[..., 2:] >> 4], dim=-1).double() - 8
        return (_f16(b[..., :2]) * q).reshape(n, k)
    if type_ == "Q8_0":
        return (_f16(b[..., :2]) * b[..., 2:].view(torch.int8).double()).reshape(n, k)
    if type_ == "Q4_K":  # eight sub-blocks of 32: 6-bit scales and minima in 12 bytes
        p = b[..., 4:16]
        sc = torch.cat([p[..., 0:4] & 63, (p[..., 8:12] & 15) | ((p[..., 0:4] >> 6) << 4)], dim=-1).double()
        mn = torch.cat([p[..., 4:8] & 63, (p[..., 8:12] >> 4) | ((p[..., 4:8] >> 6) << 4)], dim=-1).double()
        qs = b[..., 16:].reshape(n, -1, 4, 32)
        q = torch.stack([qs & 15, qs >> 4], dim=-2).reshape(n, -1, 8, 32).double()
        return ((_f16(b[..., 0:2]) * sc)[..., None] * q - (_f16(b[..., 2:4]) * mn)[..., None]).reshape(n, k)
    low, high = b[..., :128].reshape(n, -1, 2, 1, 64), b[..., 128:192].reshape(n, -1, 2, 1, 32)
    nib = torch.cat([low & 15, low >> 4], dim=-2).reshape(n, -1, 2, 4, 32)
    two = torch.cat([(high >> (2 * j)) & 3 for j in range(4)], dim=-2)
    q = (nib | (two << 4)).reshape(n, -1, 16, 16).double() - 32
    return ((_f16(b[..., 208:]) * b[..., 192:208].view(torch.int8).double())[..., None] * q).reshape(n, k)


def _mxfp4_64(blocks, scales):
    """``[rows, k]`` of one expert."""
    value = torch.tensor([0, 0.5, 1, 1.5, 2, 3, 4, 6, -0.0, -0.5, -1, -1.5, -2, -3, -4, -6], device="cuda", dtype=torch.float64)
    codes = torch.stack([blocks & 15, blocks >> 4], dim=-1).reshape(*blocks.shape[:2], 32)
    return (value[codes.long()] * torch.exp2(scales.double() - 127)[..., None]).reshape(blocks.shape[0], -1)


def _moe64(case, t):
    """Router logits are a bf16 linear's, rounded as such; all that follows them is in 64 bits."""
    x, top = t["x"].double(), case["top_k"]
    logits = (x @ t["router"].double().T + t["router_bias"].double()).to(torch.bfloat16).double()
    best, chosen = torch.sort(torch.softmax(logits, dim=-1), dim=-1, descending=True, stable=True)
    weight, chosen = best[:, :top] / best[:, :top].sum(-1, keepdim=True), chosen[:, :top]
    out = torch.zeros_like(x)
    for e in range(case["experts"]):
        token, slot = torch.nonzero(chosen == e, as_tuple=True)
        gu = x[token] @ _mxfp4_64(t["gate_up"][0][e], t["gate_up"][1][e]).T + t["gate_up_bias"][e].double()
        gate, up = gu[:, 0::2].clamp(max=7.0), gu[:, 1::2].clamp(-7.0, 7.0)
        h = (up + 1) * gate * torch.sigmoid(1.702 * gate)
        y = h @ _mxfp4_64(t["down"][0][e], t["down"][1][e]).T + t["down_bias"][e].double()
        out.index_add_(0, token, y * weight[token, slot][:, None])
    return out


def exact(case, seed):
    t, kind = _inputs(case, seed), case["kind"]
    x = t["x"].double()
    if kind == "awq_layer":
        gate, up = (t["ffn_in"].double() @ _awq64(*t["ffn"])).chunk(2, dim=-1)
        act = torch.nn.functional.silu(gate) * up
        return {"qkv": x @ _awq64(*t["qkv"]), "o": t["attn"].double() @ _awq64(*t["o"]), "ffn": act,
                "down": act @ _awq64(*t["down"])}
    if kind == "moe":
        return _moe64(case, t)
    if kind == "gptq":
        return x @ _gptq64(*t["weight"])
    if kind == "gguf":
        return x @ _gguf64(case["type"], t["weight"], case["n"], case["k"]).T
    w, scale = t["weight"]
    n, k = w.shape
    w = w.double().reshape(n // 128, 128, k // 128, 128) * scale.double()[:, None, :, None]
    return x @ w.reshape(n, k).T
