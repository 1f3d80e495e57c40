"""The grouped unpack + tcgen05 kernel of the 4-bit layouts (``oxq_packed4_matmul``): sizes at its edges.

Products of integers and bf16 values are exact, a group's sum and the totals are kept in f32: against 64-bit sums over the
exact weights a value is off by a few dozen f32 roundings of the sum of |x w| at most, so 2^-17 of that sum bounds it (plus one
bf16 rounding where y is bf16).
"""
import numpy as np
import pytest
import torch

import oracle
from oxydllm_b200 import _lib, gemm, synth
from oxydllm_b200 import linear as L

pytestmark = pytest.mark.gpu


def layer(k, n, g, gptq, seed):
    rng = np.random.default_rng(seed)
    shape_w, shape_z = ((k // 8, n), (k // g, n // 8)) if gptq else ((k, n // 8), (k // g, n // 8))
    qw, qz = (rng.integers(0, 2**32, size=s, dtype=np.uint64).astype(np.uint32) for s in (shape_w, shape_z))
    sc = (np.abs(rng.standard_normal((k // g, n)) * 0.02) / 7 + 1e-4).astype(np.float16)
    new = (lambda *a: L.QuantWeight.new_gptq(4, False, *a)) if gptq else (lambda *a: L.QuantWeight.new_awq(4, *a))
    lin = L.PackedQuantLinear(new(*(torch.from_numpy(a.view(np.int32)).cuda() for a in (qw, qz)), torch.from_numpy(sc).cuda()))
    return lin, (oracle.gptq_dequant(qw, qz, sc, 4, False) if gptq else oracle.awq_dequant(qw, qz, sc)).astype(np.float64)


def check(y, x, w):
    ref, mass = x.astype(np.float64) @ w.T, np.abs(x).astype(np.float64) @ np.abs(w).T
    rounding = 2.0**-8 * np.abs(ref) if y.dtype == torch.bfloat16 else 0.0
    assert (np.abs(y.double().cpu().numpy() - ref) <= 2.0**-17 * mass + rounding).all()


# one unit and one tile; units beyond every ring (k = 5632, shares inside their tiles); groups of 64, 128 and more; whole tiles,
# 148 of them too; one token, the edges of the tile widths and two tiles of tokens
@pytest.mark.parametrize("gptq", [False, True])
@pytest.mark.parametrize("k,n,g", [(128, 128, 64), (5632, 256, 64), (5632, 128, 512), (2048, 1152, 128), (1024, 18944, 256)])
@pytest.mark.parametrize("m", [1, 16, 17, 33, 97, 128, 129, 256])
def test_grouped_kernel_matches_64_bit_sums(cuda, m, k, n, g, gptq):
    lin, w = layer(k, n, g, gptq, seed=k + n + m)
    if m > lin._grouped_max_m:
        pytest.skip("wide layers leave the kernel earlier")
    x = synth.activations(m, k, seed=m)
    xd = torch.from_numpy(np.ascontiguousarray(x)).to(torch.bfloat16).cuda()
    y = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
    gemm.packed4_matmul(lin, xd, y)
    check(y, x, w)
    again = torch.empty_like(y)
    gemm.packed4_matmul(lin, xd, again)
    assert torch.equal(y, again)  # the parts of a shared tile are added in the order of k, not of arrival
    if m > lin.gemv_max_m():
        check(lin.forward(xd), x, w)
    gemm.check(gemm.workspace(n, k, "cuda"))


# whole tiles; two to six shares a tile, all inside it; 148 shares of 149 tiles, nearly all of which cross a tile border
@pytest.mark.parametrize("gptq", [False, True])
@pytest.mark.parametrize("k,n,g", [(1024, 1024, 128), (2048, 1024, 128), (2048, 1024, 64), (4096, 512, 64), (2048, 19072, 128)])
@pytest.mark.parametrize("m", [6, 77])
def test_shared_tiles_match_64_bit_sums(cuda, m, k, n, g, gptq):
    lin, w = layer(k, n, g, gptq, seed=k + n + m)
    if m > lin._grouped_max_m:
        pytest.skip("groups of 64 leave the kernel at 32 tokens")
    bias = torch.from_numpy(np.random.default_rng(m).standard_normal(n).astype(np.float32)).cuda()
    x = synth.activations(m, k, seed=m)
    xd = torch.from_numpy(np.ascontiguousarray(x)).to(torch.bfloat16).cuda()
    y, yb = (torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda") for _ in range(2))
    gemm.packed4_matmul(lin, xd, y)
    check(y, x, w)
    gemm.packed4_matmul(L.PackedQuantLinear(lin_raw(lin), bias), xd, yb)
    assert torch.equal(yb, y + bias)  # added to the finished sum, one f32 rounding
    gemm.check(gemm.workspace(n, k, "cuda"))


def lin_raw(lin):
    new = (lambda *a: L.QuantWeight.new_gptq(4, False, *a)) if lin.pack_dim == "in" else (lambda *a: L.QuantWeight.new_awq(4, *a))
    return new(lin.qweight, lin.qzeros, lin.scales)


@pytest.mark.parametrize("gptq", [False, True])
def test_a_replaced_tensor_is_the_one_that_counts(cuda, gptq):
    k, n, g = 256, 512, 128
    lin, _ = layer(k, n, g, gptq, seed=1)
    bias = torch.arange(n, dtype=torch.float32, device="cuda") / n
    want = L.PackedQuantLinear(lin_raw(layer(k, n, g, gptq, seed=2)[0]), bias)
    xs = [torch.from_numpy(np.ascontiguousarray(synth.activations(m, k, seed=m))).to(torch.bfloat16).cuda() for m in (1, 2, 16, 300)]
    gated, gated_want = (None if gptq else L.GatedFfnProjection(L.PackedQuantLinear(lin_raw(q))) for q in (lin, want))
    for x in xs:
        lin.forward(x)
    for one in [lin] if gptq else [lin, gated.gate_up]:
        one.qweight = want.qweight.to(torch.int64)  # as a checkpoint may hold them
        one.qzeros, one.scales = want.qzeros.t().contiguous().t(), want.scales
    lin.bias = bias
    for x in xs:
        assert torch.equal(lin.forward(x), want.forward(x))
        if not gptq:
            assert torch.equal(gated.forward(x), gated_want.forward(x))
    lin.scales = want.scales.float()  # the same values in a type that the grouped kernel does not take
    for x in xs:
        y, ref = lin.forward(x).float(), want.forward(x).float()
        assert ((y - ref).abs() <= 2e-2 * ref.abs().amax(1, keepdim=True)).all()
    lin.qweight = want.qweight.cpu()
    with pytest.raises(ValueError, match="CUDA tensors only"):
        lin.forward(xs[0])


def test_a_wait_that_ran_out_is_reported_whatever_became_of_the_workspace(cuda):
    lin, w = layer(256, 128, 128, False, seed=3)
    x = torch.from_numpy(np.ascontiguousarray(synth.activations(16, 256, seed=3))).to(torch.bfloat16).cuda()
    lin.forward(x)
    _lib.call("oxq_selftest_wait_expiry", gemm._flag_words("cuda").data_ptr(), 29, None)  # where that call's kernel reports
    ws = gemm.workspace(4096, 8192, "cuda")  # larger than a 256 x 128 layer's
    with pytest.raises(_lib.OxqError, match="bounded wait 29 .*29 = accumulator free"):
        gemm.check(ws)
    gemm.check(ws)


def test_grouped_kernel_survives_weights_that_never_come(cuda):
    ws = torch.zeros(1 << 20, dtype=torch.uint8, device="cuda")
    _lib.call("oxq_selftest_group_wait_expiry", ws.data_ptr(), ws.numel(), None)
    with pytest.raises(_lib.OxqError, match=r"bounded wait (2[1-9]|3[01]) "):
        gemm.check(ws)
    gemm.check(ws)  # reported once
    lin, w = layer(1024, 256, 128, False, seed=4)
    x = synth.activations(20, 1024, seed=4)
    check(lin.forward(torch.from_numpy(np.ascontiguousarray(x)).to(torch.bfloat16).cuda()), x, w)
    gemm.check(gemm.workspace(256, 1024, "cuda"))


def test_wide_q6k_gemv_survives_weights_that_never_come(cuda):
    scratch = torch.zeros(1 << 18, dtype=torch.uint8, device="cuda")
    _lib.call("oxq_selftest_q6k_wait_expiry", scratch.data_ptr(), scratch.numel(), None)
    with pytest.raises(_lib.OxqError, match="oxq_gguf_gemv: a bounded wait"):
        _lib.call("oxq_awq_gemv_check", None)
    _lib.call("oxq_awq_gemv_check", None)


@pytest.mark.parametrize("m", [1, 4, 12])
def test_gated_projection_into_rows_off_16_bytes(cuda, m):
    k, inter = 256, 264  # rows of 528 bytes: 16-byte pieces that all lie off a boundary once the first does
    qw, qz, sc = synth.awq_layer(k, 2 * inter, 128, seed=m)
    lin = L.PackedQuantLinear(L.QuantWeight.new_awq(4, *(torch.from_numpy(a.view(np.int32)).cuda() for a in (qw, qz)),
                                                    torch.from_numpy(sc).cuda()))
    x = torch.from_numpy(np.ascontiguousarray(synth.activations(m, k, seed=m))).to(torch.bfloat16).cuda()
    for activation in ("silu", "gelu_tanh"):
        want = L.GatedFfnProjection(lin, activation).forward(x)
        y = off16(torch.full_like(want, float("nan")), 3)
        gemm.awq_ffn_gate_up(lin, x, y, L.ACTIVATIONS[activation])
        assert torch.equal(y, want)


def off16(t, offset):
    """The same values `offset` elements behind a 16-byte boundary."""
    room = torch.zeros(t.numel() + offset, dtype=t.dtype, device=t.device)
    room[offset:] = t.reshape(-1)
    return room[offset:].view(t.shape)


@pytest.mark.parametrize("k,n", [(1024, 512), (4096, 1024), (2048, 8192)])  # GEMV up to two tokens, one, none
@pytest.mark.parametrize("m", [1, 2])
def test_gptq_decode_takes_x_on_any_4_bytes(cuda, m, k, n):
    """A row of a fused projection's output is such an x. f32 sums of products that are exact but for the scale's rounding."""
    lin, w = layer(k, n, 128, True, seed=k + m)
    x = synth.activations(m, k, seed=m)
    xd = torch.from_numpy(np.ascontiguousarray(x)).to(torch.bfloat16).cuda()
    for offset in (2, 4, 6):
        check(lin.forward(off16(xd, offset)), x, w)
    check(lin.forward(xd), x, w)


# AWQ words, zero points or scales off 16 bytes: the GEMV to 8 tokens (it wants the words aligned), then the GEMM on slabs, which
# rounds the weights to bf16 (2^-9 each) before it multiplies
@pytest.mark.parametrize("gptq", [False, True])
@pytest.mark.parametrize("m", [2, 9, 16, 17, 32])
@pytest.mark.parametrize("which", [0, 1, 2])
def test_packed_tensors_off_16_bytes(cuda, which, m, gptq):
    k, n, g = 512, 256, 128
    lin, w = layer(k, n, g, gptq, seed=m)
    tensors = [lin.qweight, lin.qzeros, lin.scales]
    tensors[which] = off16(tensors[which], 2 if which == 2 else 1)
    new = (lambda *a: L.QuantWeight.new_gptq(4, False, *a)) if gptq else (lambda *a: L.QuantWeight.new_awq(4, *a))
    odd = L.PackedQuantLinear(new(*tensors))
    x = synth.activations(m, k, seed=m)
    xd = torch.from_numpy(np.ascontiguousarray(x)).to(torch.bfloat16).cuda()
    if m == 2 and which == 0 and not gptq:
        with pytest.raises(Exception, match="16-byte aligned"):  # as ever
            odd.forward(xd)
        return
    ref, mass = x.astype(np.float64) @ w.T, np.abs(x).astype(np.float64) @ np.abs(w).T
    assert (np.abs(odd.forward(xd).double().cpu().numpy() - ref) <= 2.0**-8 * mass + 2.0**-8 * np.abs(ref)).all()


def test_calls_on_two_streams_and_a_replayed_graph_do_not_meet(cuda):
    lin, w = layer(4096, 1024, 128, False, seed=5)
    xs = [torch.from_numpy(np.ascontiguousarray(synth.activations(48, 4096, seed=s))).to(torch.bfloat16).cuda() for s in range(2)]
    want = [lin.forward(x) for x in xs]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in xs]
    got = [[], []]
    for _ in range(20):
        for i, st in enumerate(streams):
            with torch.cuda.stream(st):
                got[i].append(lin.forward(xs[i]))
    torch.cuda.synchronize()
    assert all(torch.equal(y, want[i]) for i in range(2) for y in got[i])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = lin.forward(xs[0])
    for _ in range(3):
        y.zero_()
        graph.replay()
        assert torch.equal(y, want[0])


# ------------------------------------------------------------------ the GGUF GEMV of wide layers (vocabulary projections)
# k = 14336: x of three tokens leaves room for two stages per engine, of four it does not (the narrow kernel)
@pytest.mark.parametrize("m,k,n", [(1, 2048, 9472), (3, 4096, 9480), (8, 4096, 9479), (3, 14336, 9472), (4, 14336, 9472), (8, 2048, 9472)])
def test_wide_q6k_gemv_matches_64_bit_sums(cuda, m, k, n):
    """x and the 6-bit integers are exact in f16; 16-wide sums, times d * scale (one rounding), are added in f32."""
    from oxydllm_b200 import formats as F
    data = synth.gguf_layer(F.GGML_Q6_K, 64, k, seed=k + m)
    data = np.tile(np.asarray(data).reshape(64, -1), (n // 64 + 1, 1))[:n].reshape(-1)
    w = oracle.gguf_dequant(F.GGML_Q6_K, data[: 64 * (data.size // n)], 64, k).astype(np.float64)
    bias = torch.arange(n, dtype=torch.float32, device="cuda") / n
    lin = L.QLinear(F.GGML_Q6_K, torch.from_numpy(data).cuda(), n, k, bias=bias, out_dtype=torch.float32)
    x = synth.activations(m, k, seed=m)
    y = lin.forward(torch.from_numpy(np.ascontiguousarray(x)).to(torch.bfloat16).cuda()).double().cpu().numpy()
    rows = np.arange(n) % 64
    ref, mass = (x.astype(np.float64) @ w.T)[:, rows] + bias.cpu().numpy(), (np.abs(x).astype(np.float64) @ np.abs(w).T)[:, rows] + 1
    assert (np.abs(y - ref) <= 2.0**-17 * mass).all()
    from oxydllm_b200 import _lib
    assert _lib.load().oxq_awq_gemv_check(None) == 0
