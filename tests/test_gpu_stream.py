"""The kernels that stream GGUF blocks (``oxq_gguf_matmul``) and 4-bit words (``oxq_packed4_matmul`` where ``oxq_packed4_streams``) through mma.sync or
tensor memory, at the sizes where they can go wrong, against the oracle."""
import numpy as np
import pytest
import torch

import oracle
from oxydllm_b200 import _lib, formats as F, gemm, linear as L, synth

pytestmark = pytest.mark.gpu


def random_blocks(ggml_type, n, k, seed):
    """Well-formed blocks: random codes and packed scales, block scales of about a hundredth."""
    per, size = F.GGML_BLOCK[ggml_type]
    rng = np.random.default_rng(seed)
    b = rng.integers(0, 256, (n * k // per, size), dtype=np.uint8)
    at = {F.GGML_Q4_0: [0], F.GGML_Q8_0: [0], F.GGML_Q4_K: [0, 2], F.GGML_Q6_K: [208]}[ggml_type]
    for o in at:
        b[:, o:o + 2] = (rng.uniform(-0.01, 0.01, len(b)).astype(np.float16)).view(np.uint8).reshape(-1, 2)
    return b.reshape(-1)


def run(lin, x, out_dtype=torch.bfloat16):
    m, k, n = x.shape[0], lin.in_features, lin.out_features
    y = torch.full((m, n), 9.0, dtype=out_dtype, device="cuda")
    tiles = -(-n // 128) * -(-m // 8)  # more scratch than any call of this size needs; what lies in it does not matter
    scratch = torch.randint(0, 256, (2048 * (m + 8) + tiles * 70000 + 148 * 40000,), dtype=torch.uint8, device="cuda")
    flag = gemm._flag_words(x.device)
    bp, bd = gemm._bias(lin.bias)
    _lib.call("oxq_gguf_matmul", lin.ggml_type, x.data_ptr(), _lib.OXQ_BF16, lin.blocks.data_ptr(), bp, bd, y.data_ptr(), gemm._dt(out_dtype), m, k, n,
              flag.data_ptr(), scratch.data_ptr(), scratch.numel(), gemm._st())
    gemm.check(flag)
    return y


# one unit and one tile; edges of tiles; out features that fill no tile; token blocks of 8, 16, 32, 64, and two and four of them; few tiles in many
# parts, one tile a CTA, shares across tile borders (n = 24000: 188 tiles on 148 SMs)
SIZES = [(1, 256, 2), (8, 512, 128), (9, 768, 130), (16, 2048, 256), (17, 1024, 384), (33, 2048, 126), (64, 512, 512), (65, 2048, 200), (200, 512, 1024),
         (3, 14336, 256), (5, 2048, 24000)]


@pytest.mark.parametrize("ggml_type", [F.GGML_Q4_0, F.GGML_Q8_0, F.GGML_Q4_K, F.GGML_Q6_K])
@pytest.mark.parametrize("m,k,n", SIZES)
def test_stream_matches_oracle(cuda, ggml_type, m, k, n):
    if ggml_type == F.GGML_Q6_K and k % 2048:
        pytest.skip("rows of Q6_K blocks are multiples of 16 bytes from 2048 weights on")
    data = random_blocks(ggml_type, n, k, seed=m + n)
    x = synth.activations(m, k, seed=k + m)
    bias = synth.bf16_round(np.random.default_rng(1).standard_normal(n).astype(np.float32))
    ref = oracle.linear(x, oracle.gguf_dequant(ggml_type, data, n, k), bias)
    lin = L.QLinear(ggml_type, torch.from_numpy(np.ascontiguousarray(data)).cuda(), n, k, torch.from_numpy(bias).to(torch.bfloat16).cuda())
    xc = torch.from_numpy(x).to(torch.bfloat16).cuda()
    got = run(lin, xc, torch.float32).cpu().numpy()
    # f32 sums of k products in another order: their rounding is below 2^-22 of the sum of magnitudes (Q4_K adds 128 times that of x, taken off again)
    mass = np.abs(x) @ np.abs(oracle.gguf_dequant(ggml_type, data, n, k)).T
    assert (np.abs(got - ref) <= 2.0**-15 * mass + 1e-6).all()
    assert torch.equal(run(lin, xc, torch.float32).cpu(), torch.from_numpy(got))  # the same bits again


def test_stream_infinite_and_missing_activations(cuda):
    """Infinities and NaN come out as whole weights times x give them; tokens beside them are untouched."""
    for ggml_type in (F.GGML_Q4_0, F.GGML_Q8_0, F.GGML_Q4_K, F.GGML_Q6_K):
        n, k = 130, 2048
        data = random_blocks(ggml_type, n, k, seed=3)
        x = synth.activations(3, k, seed=4)
        x[0, 5], x[1, 700] = np.inf, np.nan
        w = oracle.gguf_dequant(ggml_type, data, n, k)
        lin = L.QLinear(ggml_type, torch.from_numpy(np.ascontiguousarray(data)).cuda(), n, k)
        got = run(lin, torch.from_numpy(x).to(torch.bfloat16).cuda(), torch.float32).cpu().numpy()
        sign = w[:, 5]
        assert np.array_equal(got[0][sign != 0], np.where(sign > 0, np.inf, -np.inf)[sign != 0]) and np.isnan(got[0][sign == 0]).all()
        assert np.isnan(got[1]).all()
        ref = oracle.linear(x[2:], w)
        assert np.abs(got[2:] - ref).max() <= 1e-3 * np.abs(ref).max()


@pytest.mark.parametrize("ggml_type,m,k,n", [(F.GGML_Q4_0, 4, 4096, 4096), (F.GGML_Q8_0, 16, 2048, 6144), (F.GGML_Q4_K, 32, 4096, 4096), (F.GGML_Q6_K, 64, 14336, 1024)])
def test_operator_takes_the_stream_kernel(cuda, ggml_type, m, k, n):
    data = torch.from_numpy(random_blocks(ggml_type, n, k, seed=1)).cuda()
    lin = L.QLinear(ggml_type, data, n, k)
    x = torch.from_numpy(synth.activations(m, k, seed=2)).to(torch.bfloat16).cuda()
    assert _lib.entry("oxq_gguf_scratch_bytes")(ggml_type, m, k, n) > 0
    assert torch.equal(lin.forward(x), run(lin, x))
    off = torch.empty(m * k + 4, dtype=torch.bfloat16, device="cuda")[4:].view(m, k).copy_(x)  # on 8 bytes only: the other kernels
    if m <= 32:
        assert (lin.forward(off).float() - lin.forward(x).float()).abs().max() <= 2e-2 * lin.forward(x).float().abs().max()


def test_scratch_that_is_too_small_is_refused(cuda):
    n = k = 4096
    lin = L.QLinear(F.GGML_Q4_0, torch.zeros(n * k // 32 * 18, dtype=torch.uint8, device="cuda"), n, k)
    x = torch.zeros(4, k, dtype=torch.bfloat16, device="cuda")
    y = torch.empty(4, n, dtype=torch.bfloat16, device="cuda")
    need = _lib.entry("oxq_gguf_scratch_bytes")(lin.ggml_type, 4, k, n)
    scratch = torch.empty(need, dtype=torch.uint8, device="cuda")
    with pytest.raises(_lib.OxqError):
        _lib.call("oxq_gguf_matmul", lin.ggml_type, x.data_ptr(), _lib.OXQ_BF16, lin.blocks.data_ptr(), 0, 0, y.data_ptr(), _lib.OXQ_BF16, 4, k, n,
                  gemm._flag_words(x.device).data_ptr(), scratch.data_ptr(), need - 256, gemm._st())


def packed_layer(fmt, k, n, g, seed, bias=None):
    """An AWQ ("awq") or GPTQ ("gptq", symmetric "sym") layer of random words and its weights [n, k] in 64 bits."""
    rng = np.random.default_rng(seed)
    words = lambda *shape: rng.integers(0, 2**32, shape, dtype=np.uint64).astype(np.uint32)
    qw, qz = words(*((k, n // 8) if fmt == "awq" else (k // 8, n))), words(k // g, n // 8)
    sc = rng.uniform(-0.02, 0.02, (k // g, n)).astype(np.float16)
    dev = [torch.from_numpy(a.view(np.int32)).cuda() for a in (qw, qz)] + [torch.from_numpy(sc).cuda()]
    raw = L.QuantWeight.new_awq(4, *dev) if fmt == "awq" else L.QuantWeight.new_gptq(4, fmt == "sym", *dev)
    w = oracle.awq_dequant(qw, qz, sc) if fmt == "awq" else oracle.gptq_dequant(qw, qz, sc, 4, fmt == "sym")
    return L.PackedQuantLinear(raw, bias), w.astype(np.float64)


def packed(lin, x, out_dtype=torch.float32):
    y = torch.full((x.shape[0], lin.out_features), 9.0, dtype=out_dtype, device="cuda")
    gemm.packed4_matmul(lin, x, y)
    gemm.check(gemm._flag_words(x.device))
    return y


# one unit and one tile; half a tile (n = 128, 384, 896); groups of 32, 64, 128, 256 and more; token blocks of 8 and 16, and two to four of them; few tiles in many
# parts, shares across tile borders (n = 20480: 80 tiles on 148 SMs; 37888: 148 tiles)
PACKED_SIZES = [("gptq", 1, 2048, 128, 32), ("gptq", 4, 128, 128, 128), ("gptq", 3, 1024, 384, 64), ("sym", 8, 4096, 896, 128), ("gptq", 9, 4096, 1152, 32), ("sym", 33, 4096, 128, 32),
                ("gptq", 16, 2048, 37888, 64), ("gptq", 5, 4096, 512, 1024), ("sym", 2, 14336, 1024, 256), ("gptq", 16, 4096, 20480, 128),
                ("awq", 1, 5632, 128, 128), ("awq", 8, 5632, 384, 128), ("awq", 3, 5632, 256, 512), ("awq", 8, 14336, 896, 64), ("awq", 9, 2048, 512, 32), ("awq", 17, 4096, 384, 32),
                ("awq", 1, 7168, 128, 32), ("awq", 16, 4096, 20480, 128), ("awq", 12, 8192, 3584, 64), ("awq", 7, 2048, 37888, 128)]

# through tensor memory: half a tile; every width of a tile of tokens and its edges; two and three blocks of tokens; groups of 32 to 1024; whole tiles, one
# a CTA (n = 37888); clusters of two (n = 16384), five (6144) and eight; shares across tile borders (n = 38144: 149 tiles)
WIDE_SIZES = [("awq", 9, 1024, 128, 128), ("awq", 16, 1024, 256, 64), ("awq", 17, 1024, 384, 128), ("awq", 32, 2048, 640, 64), ("awq", 33, 1024, 128, 32), ("awq", 48, 4096, 6144, 256),
              ("awq", 64, 3072, 16384, 64), ("awq", 65, 2048, 384, 1024), ("awq", 80, 2048, 37888, 128), ("awq", 96, 4096, 1024, 32), ("awq", 97, 2048, 1280, 64), ("awq", 192, 1024, 896, 128),
              ("awq", 193, 2048, 384, 128), ("awq", 256, 1024, 640, 64), ("awq", 17, 2048, 38144, 128), ("awq", 96, 1024, 38144, 64), ("awq", 3, 2048, 11264, 128),
              ("gptq", 3, 2048, 128, 128), ("gptq", 9, 1024, 384, 128), ("sym", 31, 2048, 1152, 64), ("gptq", 49, 1024, 2048, 32), ("gptq", 77, 2048, 6144, 128), ("sym", 95, 14336, 128, 512),
              ("gptq", 112, 2048, 1024, 64), ("gptq", 40, 3072, 38144, 128), ("gptq", 20, 8192, 2048, 256)]


@pytest.mark.parametrize("fmt,m,k,n,g", PACKED_SIZES + WIDE_SIZES)
def test_packed_stream_matches_oracle(cuda, fmt, m, k, n, g):
    assert _lib.entry("oxq_packed4_streams")(m, k, n, g, int(fmt != "awq")) == 1
    x, bias = synth.activations(m, k, seed=k + m), synth.bf16_round(np.random.default_rng(1).standard_normal(n).astype(np.float32))
    lin, w = packed_layer(fmt, k, n, g, m + n, torch.from_numpy(bias).to(torch.bfloat16).cuda())
    xc = torch.from_numpy(np.ascontiguousarray(x)).to(torch.bfloat16).cuda()
    got = packed(lin, xc)
    # products of small integers and bf16 values are exact; the f32 sums of k of them are off by less than 2^-17 of the sum of magnitudes
    ref, mass = x.astype(np.float64) @ w.T + bias, np.abs(x).astype(np.float64) @ np.abs(w).T + np.abs(bias)
    assert (np.abs(got.double().cpu().numpy() - ref) <= 2.0**-17 * mass + 1e-6).all()
    assert torch.equal(packed(lin, xc), got)  # the same bits again
    y = lin.forward(xc)
    assert lin._streams(m) and torch.equal(y, got.to(torch.bfloat16))  # what the layer takes


def test_packed_stream_infinite_and_missing_activations(cuda):
    for fmt, k, n, g, m in (("awq", 5632, 384, 128, 3), ("gptq", 16384, 384, 64, 3), ("sym", 4096, 384, 32, 3), ("awq", 2048, 384, 64, 40), ("gptq", 2048, 384, 32, 70)):
        lin, w = packed_layer(fmt, k, n, g, 3)
        x = synth.activations(m, k, seed=4)
        x[0, 5], x[1, 700] = np.inf, np.nan
        got = packed(lin, torch.from_numpy(x).to(torch.bfloat16).cuda()).cpu().numpy()
        sign = np.sign(w[:, 5])
        assert np.array_equal(got[0][sign != 0], np.where(sign > 0, np.inf, -np.inf)[sign != 0]) and np.isnan(got[0][sign == 0]).all()
        assert np.isnan(got[1]).all()
        ref, mass = x[2:].astype(np.float64) @ w.T, np.abs(x[2:]).astype(np.float64) @ np.abs(w).T
        assert (np.abs(got[2:] - ref) <= 2.0**-17 * mass + 1e-6).all()


@pytest.mark.parametrize("act", ["silu", "gelu_tanh"])
@pytest.mark.parametrize("m,k,inter,g", [(1, 5632, 128, 128), (8, 5632, 1152, 64), (16, 4096, 10240, 128), (33, 4096, 640, 32), (7, 2048, 18944, 128), (9, 2048, 640, 64), (20, 2048, 18944, 128),
                                       (96, 1024, 19072, 128), (33, 1024, 19072, 64), (150, 2048, 384, 128)])
def test_gate_and_up_meet_in_one_tile(cuda, m, k, inter, g, act):
    assert _lib.entry("oxq_packed4_streams")(m, k, 2 * inter, g, 0) == 1
    lin, w = packed_layer("awq", k, 2 * inter, g, m + inter)
    x = synth.activations(m, k, seed=m)
    xc = torch.from_numpy(np.ascontiguousarray(x)).to(torch.bfloat16).cuda()
    y = L.GatedFfnProjection(lin, act).forward(xc)
    gate, up = (torch.from_numpy(x.astype(np.float64) @ w[i * inter:(i + 1) * inter].T) for i in (0, 1))
    f = torch.nn.functional.silu(gate) if act == "silu" else torch.nn.functional.gelu(gate, approximate="tanh")
    # one bf16 rounding, and sums that are off by 2^-17 of their magnitudes in a function whose slope is at most 1.13
    mass = [torch.from_numpy(np.abs(x).astype(np.float64) @ np.abs(w[i * inter:(i + 1) * inter]).T) * 2.0**-17 for i in (0, 1)]
    bound = 2.0**-8 * (f * up).abs() + 1.13 * mass[0] * up.abs() + mass[1] * (f.abs() + mass[0]) + 2.0**-18 * (f * up).abs() + 1e-6
    assert ((y.double().cpu() - f * up).abs() <= bound).all()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        again = L.GatedFfnProjection(lin, act).forward(xc)
    for _ in range(3):  # marks of an earlier replay are not taken for this one's
        again.fill_(9.0)
        graph.replay()
        assert torch.equal(again, y)


def test_wide_kernel_takes_bf16_scales(cuda):
    k, n, g, m = 2048, 640, 64, 20
    rng = np.random.default_rng(5)
    qw, qz = (rng.integers(0, 2**32, shape, dtype=np.uint64).astype(np.uint32) for shape in ((k, n // 8), (k // g, n // 8)))
    sc = synth.bf16_round(rng.uniform(0.001, 0.02, (k // g, n)).astype(np.float32))
    lin = L.PackedQuantLinear(L.QuantWeight.new_awq(4, *(torch.from_numpy(a.view(np.int32)).cuda() for a in (qw, qz)), torch.from_numpy(sc).to(torch.bfloat16).cuda()))
    x = synth.activations(m, k, seed=1)
    w = oracle.awq_dequant(qw, qz, np.ones_like(sc, dtype=np.float16)).astype(np.float64) * np.repeat(sc.astype(np.float64), g, axis=0).T
    got = packed(lin, torch.from_numpy(np.ascontiguousarray(x)).to(torch.bfloat16).cuda()).double().cpu().numpy()
    assert (np.abs(got - x.astype(np.float64) @ w.T) <= 2.0**-17 * (np.abs(x).astype(np.float64) @ np.abs(w).T) + 1e-6).all()
