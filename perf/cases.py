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
    return PackedQuantLinear(QuantWeight.new_awq(4, _words(g, k, n // 8), _words(g, k // group, n // 8),
                                                 _scales(g, k // group, n)))


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


def prepare(case, seed):
    g = _gen(seed)
    m, kind = case["tokens"], case["kind"]
    if kind == "awq_layer":
        h, i, grp = case["hidden"], case["inter"], case["group"]
        return {"kind": kind, "x": _x(g, m, h), "attn": _x(g, m, h), "ffn_in": _x(g, m, h),
                "qkv": _awq(g, h, h + 2 * case["kv"], grp), "o": _awq(g, h, h, grp),
                "ffn": GatedFfnProjection(_awq(g, h, 2 * i, grp), "silu"), "down": _awq(g, i, h, grp)}
    if kind == "moe":
        e, h, i = case["experts"], case["hidden"], case["inter"]
        gu_b, gu_s = _mxfp4_experts(g, e, 2 * i, h)
        dn_b, dn_s = _mxfp4_experts(g, e, h, i)
        small = lambda *shape: (torch.randn(*shape, generator=g, device="cuda") * 0.02).to(torch.bfloat16)  # noqa: E731
        layer = GptOssMoe(gu_b, gu_s, small(e, 2 * i), dn_b, dn_s, small(e, h), h, i, top_k=case["top_k"],
                          router_weight=small(e, h), router_bias=small(e))
        return {"kind": kind, "x": _x(g, m, h), "layer": layer}
    k, n = case["k"], case["n"]
    if kind == "gptq":
        zeros = None if case["sym"] else _words(g, k // case["group"], n // 8)
        layer = PackedQuantLinear(QuantWeight.new_gptq(4, case["sym"], _words(g, k // 8, n), zeros,
                                                       _scales(g, k // case["group"], n)))
    elif kind == "gguf":
        layer = QLinear(GGUF_TYPES[case["type"]], _gguf_blocks(g, case["type"], n, k), n, k)
    else:
        w = torch.randn(n // 128, 128, k // 128, 128, generator=g, device="cuda") * 0.02
        scale = w.abs().amax(dim=(1, 3)) / 448.0
        w = (w / scale[:, None, :, None]).clamp(-448.0, 448.0).reshape(n, k).to(torch.float8_e4m3fn)
        layer = Fp8Linear(w, scale)
    return {"kind": kind, "x": _x(g, m, k), "layer": layer}


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
