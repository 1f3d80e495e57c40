"""The kernel that streams GGUF blocks through mma.sync (``oxq_gguf_matmul``), at the sizes where it can go wrong, against the oracle."""
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
