"""The block-scaled tensor-core kernels (MXFP4 experts of small batches): sizes at their edges.

Weights are operands as stored and a bf16 activation is the sum of two E4M3 pieces, exact but for 2^-21 of the largest of its block
of 32; products are exact and sums are f32. Against 64-bit sums over the exact weights a value is off by a few dozen f32 roundings
of the sum of |x w| at most, so 2^-17 of that sum bounds it, plus one bf16 rounding of the result.
"""
import numpy as np
import pytest
import torch

import oracle
from oxydllm_b200 import _lib, gemm, synth

pytestmark = pytest.mark.gpu


def bf16(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(torch.bfloat16).cuda()


# ------------------------------------------------------------------------------------------------------- MXFP4 experts, small batches
def experts_layer(experts, hidden, inter, seed):
    from oxydllm_b200 import moe
    d = synth.gptoss_moe(experts, hidden, inter, 1, seed=seed)
    t = lambda a, dt=None: torch.from_numpy(np.ascontiguousarray(a)).to(dt or torch.uint8).cuda()  # noqa: E731
    layer = moe.GptOssMoe(t(d["gu_blocks"]), t(d["gu_scales"]), t(d["gu_bias"], torch.bfloat16), t(d["dn_blocks"]), t(d["dn_scales"]),
                          t(d["dn_bias"], torch.bfloat16), hidden=hidden, inter=inter, top_k=4)
    return layer, d


# rows per expert around a token block and its columns (16, 48), experts without rows; one stage, stages that end after 1, 2 and 3
# blocks of 32, scale rows of odd, even and whole-word lengths; feature tiles that end inside
@pytest.mark.parametrize("hidden,inter", [(32, 96), (96, 32), (160, 224), (2880, 64), (384, 2880), (256, 512)])
@pytest.mark.parametrize("counts", [(70, 0, 1, 0), (16, 17, 48, 49), (0, 0, 0, 100), (47, 64, 15, 33)])
def test_moe_small_batch_matches_64_bit_experts(cuda, hidden, inter, counts):
    layer, d = experts_layer(len(counts), hidden, inter, seed=hidden + inter)
    ids = np.random.default_rng(1).permutation(np.repeat(np.arange(len(counts)), counts))
    x = synth.activations(len(ids), hidden, seed=len(ids))
    y = layer.forward_experts(bf16(x), torch.from_numpy(ids).cuda())
    layer.check()
    got = y.double().cpu().numpy()
    gb, db = (b.double().cpu().numpy() for b in (layer.gu_bias, layer.dn_bias))
    for e, c in enumerate(counts):
        rows = np.nonzero(ids == e)[0]
        gu = oracle.mxfp4_dequant(d["gu_blocks"][e], d["gu_scales"][e], 2 * inter, hidden).astype(np.float64)
        dn = oracle.mxfp4_dequant(d["dn_blocks"][e], d["dn_scales"][e], hidden, inter).astype(np.float64)
        a = x[rows].astype(np.float64) @ gu.T + gb[e]
        gate, up = np.minimum(a[:, 0::2], 7.0), np.clip(a[:, 1::2], -7.0, 7.0)
        h = (up + 1) * gate / (1 + np.exp(-1.702 * gate))
        ref = h @ dn.T + db[e]
        # h is rounded to bf16 (2^-9 of each), as is the result; sums and the activation are good to some 2^-17
        assert (np.abs(got[rows] - ref) <= 2.0**-8 * (np.abs(h) @ np.abs(dn).T + np.abs(ref)) + 1e-6).all(), (e, c)


def test_moe_small_batch_kernel_survives_weights_that_never_come(cuda):
    ws = torch.zeros(1 << 20, dtype=torch.uint8, device="cuda")
    _lib.call("oxq_selftest_moe_mx_wait_expiry", ws.data_ptr(), ws.numel(), None)
    with pytest.raises(_lib.OxqError, match=r"bounded wait 6[1-7] "):
        gemm.check(ws)
    gemm.check(ws)  # reported once
    test_moe_small_batch_matches_64_bit_experts(cuda, 256, 512, (16, 17, 48, 49))

