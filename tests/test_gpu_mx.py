"""The block-scaled tensor-core kernels (E4M3 weights, MXFP4 experts of small batches): sizes at their edges.

Weights are operands as stored and a bf16 activation is the sum of two E4M3 pieces, exact but for 2^-21 of the largest of its block
of 32, or of four, exact but for 2^-34, where half of the block is small beside its largest; products are exact and sums are f32. Against 64-bit sums over the exact weights a value is off by a few dozen f32 roundings
of the sum of |x w| at most, so 2^-17 of that sum bounds it, plus one bf16 rounding of the result.
"""
import numpy as np
import pytest
import torch

import oracle
from oxydllm_b200 import _lib, gemm, synth
from oxydllm_b200 import linear as L

pytestmark = pytest.mark.gpu


def bf16(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(torch.bfloat16).cuda()


def fp8_weights(n, k, s_out, s_in, seed):
    rng = np.random.default_rng(seed)
    w8 = rng.integers(0, 256, (n, k), dtype=np.uint8)
    w8[(w8 & 0x7F) == 0x7F] = 0x08  # no NaN
    scale = (rng.random((s_out, s_in)) * 0.01 + 1e-3).astype(np.float32)
    full = np.repeat(np.repeat(scale.astype(np.float64), n // s_out, 0), k // s_in, 1)
    return w8, scale, oracle.fp8_dequant(w8, None).astype(np.float64) * full


def fp8_gemm(w8, scale, xd, n, k, bias=None):
    m = xd.shape[0]
    ws = gemm.workspace(n, k, "cuda")
    y = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
    wd, sd = torch.from_numpy(w8).cuda(), None if scale is None else torch.from_numpy(scale).cuda()
    s_out, s_in = (0, 0) if scale is None else scale.shape
    _lib.call("oxq_fp8_gemm", xd.data_ptr(), _lib.OXQ_BF16, wd.data_ptr(), 0 if sd is None else sd.data_ptr(), s_out, s_in,
              0 if bias is None else bias.data_ptr(), _lib.OXQ_F32, y.data_ptr(), _lib.OXQ_F32, m, k, n, ws.data_ptr(), ws.numel(), None)
    gemm.check(ws)
    return y


def close(y, x, w, extra=0.0):
    ref, mass = x.astype(np.float64) @ w.T, np.abs(x).astype(np.float64) @ np.abs(w).T
    assert (np.abs(y.double().cpu().numpy() - ref) <= 2.0**-17 * mass + extra).all()


# one unit and one tile; blocks of 64 columns (two folds a unit) and of 192 rows' worth; whole rows; 148 tiles and more
@pytest.mark.parametrize("n,k,s_out,s_in", [(128, 128, 1, 1), (256, 512, 1, 8), (384, 1536, 3, 8), (2048, 512, 16, 4), (19072, 256, 149, 2)])
@pytest.mark.parametrize("m", [1, 16, 17, 33, 64, 65, 97, 129, 512])
def test_fp8_block_scaled_matches_64_bit_sums(cuda, m, n, k, s_out, s_in):
    w8, scale, w = fp8_weights(n, k, s_out, s_in, seed=m + n)
    x = synth.activations(m, k, seed=m)
    y = fp8_gemm(w8, scale, bf16(x), n, k)
    close(y, x, w)
    assert torch.equal(y, fp8_gemm(w8, scale, bf16(x), n, k))  # parts of a shared tile are added in the order of k


def test_fp8_block_scaled_bias_and_no_scale(cuda):
    n, k, m = 256, 256, 40
    w8, _, _ = fp8_weights(n, k, 1, 1, seed=1)
    x = synth.activations(m, k, seed=2)
    y = fp8_gemm(w8, None, bf16(x), n, k)
    close(y, x, oracle.fp8_dequant(w8, None).astype(np.float64))
    bias = torch.arange(n, dtype=torch.float32, device="cuda")
    assert torch.equal(fp8_gemm(w8, None, bf16(x), n, k, bias), y + bias)


def test_fp8_block_scaled_activations_of_every_magnitude(cuda):
    """Outliers inside a block of 32, tokens far apart in size, zeros, subnormal scales: the pieces are exact or 2^-21 of the block's largest."""
    n, k, m = 128, 256, 40
    w8, scale, w = fp8_weights(n, k, 1, 2, seed=3)
    x = synth.activations(m, k, seed=4)
    x[1] *= 1e-30
    x[2] *= 1e30
    x[3, ::7] *= 3000.0
    x[4, :128] = 0.0
    x[5] = 0.0
    x[6] = 2.0**-120
    x[7, 5] = 1e4
    x = synth.bf16_round(x)
    y = fp8_gemm(w8, scale, bf16(x), n, k)
    block = np.repeat(np.abs(x).reshape(m, -1, 32).max(-1), 32, -1).astype(np.float64)
    close(y, x, w, extra=2.0**-20 * block @ np.abs(w).T)


def test_fp8_block_scaled_special_values_stay_special(cuda):
    n, k, m = 128, 256, 20
    w8, scale, w = fp8_weights(n, k, 1, 2, seed=5)
    w8[3, 7] = 0x7F
    x = synth.activations(m, k, seed=6)
    x[2, 9], x[4, 200] = np.inf, np.nan
    y = fp8_gemm(w8, scale, bf16(x), n, k).cpu().numpy()
    assert np.isnan(y[:, 3]).all() and not np.isfinite(y[2]).any() and np.isnan(y[4]).all()
    rows, cols = [r for r in range(m) if r not in (2, 4)], [c for c in range(n) if c != 3]
    assert np.isfinite(y[np.ix_(rows, cols)]).all()


# folds of 64 and of 128 columns; merged pieces, two MMAs, several token blocks; scratch from the least that is taken (the pieces, their
# block scales and which units have a second pair) to all that helps
@pytest.mark.parametrize("m,n,k,s_out,s_in", [(512, 512, 1024, 4, 16), (512, 512, 1024, 4, 8), (20, 256, 512, 2, 8), (65, 128, 256, 1, 4)])
def test_fp8_block_scaled_stays_inside_its_scratch(cuda, m, n, k, s_out, s_in):
    w8, scale, w = fp8_weights(n, k, s_out, s_in, seed=m)
    x = synth.activations(m, k, seed=m)
    xd, wd, sd = bf16(x), torch.from_numpy(w8).cuda(), torch.from_numpy(scale).cuda()
    blocks = -(-m // 128)
    mpad = -(-(-(-m // blocks)) // 16) * 16
    up = lambda v: -(-v // 256) * 256  # noqa: E731
    least = up(4 * blocks * mpad * k) + 2 * (k // 128 * blocks * (512 if mpad <= 32 else 1024)) + up(8 + 8 * (k // 128) * blocks)
    full = int(_lib.load().oxq_fp8_scratch_bytes(m, k, n, s_out, s_in))
    assert least < full
    for size in sorted({least, least + 256, least + (full - least) // 3, full, min(full, 1105920)}):
        if size < least:
            continue
        room = torch.full((256 + full + (1 << 20),), 0xA5, dtype=torch.uint8, device="cuda")
        room[:256] = 0
        y = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
        args = (xd.data_ptr(), _lib.OXQ_BF16, wd.data_ptr(), sd.data_ptr(), s_out, s_in, 0, _lib.OXQ_F32, y.data_ptr(), _lib.OXQ_F32, m, k, n)
        _lib.call("oxq_fp8_matmul", *args, room.data_ptr(), room.data_ptr() + 256, size, None)
        gemm.check(room)
        close(y, x, w)
        assert (room[256 + size:] == 0xA5).all()
        if 256 + size >= int(_lib.load().oxq_gemm_workspace_bytes(n, k)):  # the same kernel inside a workspace
            room[256:] = 0xA5
            _lib.call("oxq_fp8_gemm", *args, room.data_ptr(), 256 + size, None)
            gemm.check(room)
            assert (room[256 + size:] == 0xA5).all()


def activations_with_outliers(m, k, seed):
    """Values about 0.01 with 3e3 in each block of 32 (rows 0, 4, ...), with 1e4 in two columns (rows 1, 5, ...), with -1e6 in one (rows 2, 6,
    ...), rows of ordinary values; and the columns of the outliers."""
    x = 0.01 * synth.activations(m, k, seed=seed)
    x[0::4, 5::32] = 3e3
    x[1::4, [7, k // 2 + 9]] = 1e4
    x[2::4, k - 20] = -1e6
    x[3::4] *= 100.0
    return synth.bf16_round(x), np.r_[5:k:32, 7, k // 2 + 9, k - 20]


def outlier_bound(x, w):
    """What f32 sums leave of 64-bit ones, and the activations' error."""
    m, k = x.shape
    block = np.repeat(np.abs(x).reshape(m, -1, 32).max(-1), 32, -1).astype(np.float64)
    return 2.0**-17 * np.abs(x).astype(np.float64) @ np.abs(w).T + 2.0**-34 * block @ np.abs(w).T


def special_activations(m, k, seed):
    """Rows with one infinity, with two of both signs, with a NaN, others with an outlier, the rest ordinary."""
    x, _ = activations_with_outliers(m, k, seed)
    x[1, 40], x[2, [3, k - 1]], x[4, k // 2], x[5, [0, 1]] = np.inf, [np.inf, -np.inf], np.nan, -np.inf
    return x, [r for r in range(m) if r not in (1, 2, 4, 5)]


def same_special(y, x, w):
    """Where 64-bit products and sums are infinite or NaN (an infinity times zero is), these are."""
    with np.errstate(invalid="ignore"):
        ref = x.astype(np.float64) @ w.T
    for r in np.nonzero(~np.isfinite(x).all(1))[0]:
        with np.errstate(invalid="ignore"):
            p = x[r].astype(np.float64) * w
        ref[r] = [np.nan if np.isnan(q).any() or (np.isposinf(q).any() and np.isneginf(q).any()) else
                  np.inf if np.isposinf(q).any() else -np.inf if np.isneginf(q).any() else v for q, v in zip(p, ref[r])]
    assert np.array_equal(np.isnan(y), np.isnan(ref))
    assert np.array_equal(np.where(np.isinf(y), np.sign(y), 0), np.where(np.isinf(ref), np.sign(ref), 0))


# folds of 128 and of 64 columns; merged pieces, two MMAs, several token blocks; whole tiles, shares inside tiles and across them
@pytest.mark.parametrize("n,k,s_out,s_in", [(128, 128, 1, 1), (256, 1536, 2, 24), (19072, 256, 149, 2), (128, 4224, 1, 33)])
@pytest.mark.parametrize("m", [9, 20, 65, 300])
def test_fp8_zero_weights_beside_outliers(cuda, m, n, k, s_out, s_in):
    w8, scale, w = fp8_weights(n, k, s_out, s_in, seed=m + k)
    x, columns = activations_with_outliers(m, k, seed=m)
    w8[1::2, columns], w[1::2, columns] = 0, 0.0
    y = fp8_gemm(w8, scale, bf16(x), n, k)
    assert (np.abs(y.double().cpu().numpy() - x.astype(np.float64) @ w.T) <= outlier_bound(x, w)).all()
    assert torch.equal(y, fp8_gemm(w8, scale, bf16(x), n, k))


@pytest.mark.parametrize("n,k,s_out,s_in", [(128, 256, 1, 4), (512, 1024, 4, 8)])
@pytest.mark.parametrize("m", [9, 33, 140])
def test_fp8_infinities(cuda, m, n, k, s_out, s_in):
    w8, scale, w = fp8_weights(n, k, s_out, s_in, seed=m)
    w8[::5, 40], w[::5, 40] = 0, 0.0
    x, rest = special_activations(m, k, seed=m)
    y = fp8_gemm(w8, scale, bf16(x), n, k).double().cpu().numpy()
    same_special(y, x, w)
    block = np.repeat(np.abs(x[rest]).reshape(len(rest), -1, 32).max(-1), 32, -1).astype(np.float64)
    assert (np.abs(y[rest] - x[rest].astype(np.float64) @ w.T) <= outlier_bound(x[rest], w) + 2.0**-26 * block @ np.abs(w).T).all()


@pytest.mark.parametrize("m", [9, 16])
def test_fp8_decode_takes_x_on_any_8_bytes(cuda, m):
    n, k = 256, 512
    w8, scale, w = fp8_weights(n, k, 2, 4, seed=m)
    lin = L.Fp8Linear(torch.from_numpy(w8).cuda(), torch.from_numpy(scale).cuda())
    x = synth.activations(m, k, seed=m)
    room = torch.zeros(m * k + 4, dtype=torch.bfloat16, device="cuda")
    room[4:] = bf16(x).reshape(-1)
    ref = x.astype(np.float64) @ w.T
    for xd in (bf16(x), room[4:].view(m, k)):
        close(lin.forward(xd), x, w, extra=2.0**-8 * np.abs(ref))


def test_fp8_block_scaled_kernel_survives_weights_that_never_come(cuda):
    ws = torch.zeros(1 << 20, dtype=torch.uint8, device="cuda")
    _lib.call("oxq_selftest_packed_mx_wait_expiry", ws.data_ptr(), ws.numel(), None)
    with pytest.raises(_lib.OxqError, match=r"bounded wait (4[1-9]|5[01]) "):
        gemm.check(ws)
    gemm.check(ws)  # reported once
    w8, scale, w = fp8_weights(128, 128, 1, 1, seed=7)
    x = synth.activations(20, 128, seed=8)
    close(fp8_gemm(w8, scale, bf16(x), 128, 128), x, w)


# --------------------------------------------------------------------------------------------------------------- GPTQ, few tokens
# large layers of groups of 128 and more: whole tiles and shares across their borders (288 and 65 tiles), shares inside tiles (24)
@pytest.mark.parametrize("k,n,g,sym", [(1152, 36864, 128, False), (1152, 36864, 128, True), (14336, 3072, 512, False), (5120, 8320, 1024, False)])
@pytest.mark.parametrize("m", [1, 3, 15, 16])
def test_gptq_few_tokens_match_64_bit_sums(cuda, m, k, n, g, sym):
    rng = np.random.default_rng(k + m)
    qw, qz = (rng.integers(0, 2**32, size=s, dtype=np.uint64).astype(np.uint32) for s in ((k // 8, n), (k // g, n // 8)))
    sc = (np.abs(rng.standard_normal((k // g, n)) * 0.02) / 7 + 1e-4).astype(np.float16)
    dev = [torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda() for a in (qw, qz, sc)]
    lin = L.PackedQuantLinear(L.QuantWeight.new_gptq(4, sym, dev[0], None if sym else dev[1], dev[2]))
    codes = (torch.from_numpy(qw.view(np.int32)).cuda()[:, None] >> torch.arange(0, 32, 4, device="cuda", dtype=torch.int32)[None, :, None]) & 15
    zeros = 8 if sym else ((dev[1][:, :, None] >> torch.arange(0, 32, 4, device="cuda", dtype=torch.int32)) & 15).reshape(k // g, 1, n) + 1
    w = ((codes.reshape(k // g, g, n) - zeros) * dev[2].double()[:, None]).reshape(k, n)
    x = bf16(synth.activations(m, k, seed=m))
    y = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
    gemm.packed4_matmul(lin, x, y)
    ref, mass = x.double() @ w, x.double().abs() @ w.abs()
    assert ((y.double() - ref).abs() <= 2.0**-17 * mass).all()
    again = torch.empty_like(y)
    gemm.packed4_matmul(lin, x, again)
    assert torch.equal(y, again)
    if lin.gemv_max_m() < m:
        assert ((lin.forward(x).double() - ref).abs() <= 2.0**-17 * mass + 2.0**-8 * ref.abs()).all()
    gemm.check(gemm.workspace(n, k, "cuda"))


@pytest.mark.parametrize("sym", [False, True])
def test_gptq_zero_weights_beside_large_activations(cuda, sym):
    """Products with q = z are exact zeros: eight x of 8000 in every group of 128 leave nothing in the sums of the others (1 to 2 in
    magnitude, so that both pieces are exact), whose f32 roundings stay below 2^-19 of the sum of |x w|."""
    k, n, g, m = 1152, 36864, 128, 16
    rng = np.random.default_rng(k)
    x = (rng.uniform(1, 2, (m, k)) * rng.choice([-1, 1], (m, k))).astype(np.float32)
    nib = rng.integers(0, 16, (k, n), dtype=np.uint32)
    zero = np.full((k // g, n), 8, np.uint32) if sym else rng.integers(1, 16, (k // g, n), dtype=np.uint32)
    x[:, ::16] = 8000.0
    nib[::16] = np.repeat(zero, g // 16, 0)
    qw = (nib.reshape(k // 8, 8, n) << (4 * np.arange(8, dtype=np.uint32))[None, :, None]).sum(1, dtype=np.uint32)
    qz = ((zero - 1).reshape(k // g, n // 8, 8) << (4 * np.arange(8, dtype=np.uint32))).sum(2, dtype=np.uint32)
    sc = (np.abs(rng.standard_normal((k // g, n)) * 0.02) / 7 + 1e-4).astype(np.float16)
    dev = [torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda() for a in (qw, qz, sc)]
    lin = L.PackedQuantLinear(L.QuantWeight.new_gptq(4, sym, dev[0], None if sym else dev[1], dev[2]))
    y = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
    xd = bf16(x)
    gemm.packed4_matmul(lin, xd, y)
    codes = torch.from_numpy(nib.astype(np.int32)).cuda() - torch.from_numpy(np.repeat(zero, g, 0).astype(np.int32)).cuda()
    w = codes.double() * dev[2].double().repeat_interleave(g, 0)
    xd = xd.double()
    assert ((y.double() - xd @ w).abs() <= 2.0**-19 * (xd.abs() @ w.abs())).all()


@pytest.mark.parametrize("k,n,g,sym", [(1152, 36864, 128, True), (14336, 3072, 512, False)])
@pytest.mark.parametrize("special", [False, True])
def test_gptq_outliers_and_infinities(cuda, k, n, g, sym, special):
    m = 16
    rng = np.random.default_rng(k)
    x, columns = activations_with_outliers(m, k, seed=k)
    rest = list(range(m))
    if special:
        x, rest = special_activations(m, k, seed=k)
    nib = rng.integers(0, 16, (k, n), dtype=np.uint32)
    zero = np.full((k // g, n), 8, np.uint32) if sym else rng.integers(1, 16, (k // g, n), dtype=np.uint32)
    nib[columns, 1::2] = zero[columns // g, 1::2]
    nib[40, ::3] = zero[0, ::3]
    qw = (nib.reshape(k // 8, 8, n) << (4 * np.arange(8, dtype=np.uint32))[None, :, None]).sum(1, dtype=np.uint32)
    qz = ((zero - 1).reshape(k // g, n // 8, 8) << (4 * np.arange(8, dtype=np.uint32))).sum(2, dtype=np.uint32)
    sc = (np.abs(rng.standard_normal((k // g, n)) * 0.02) / 7 + 1e-4).astype(np.float16)
    dev = [torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda() for a in (qw, qz, sc)]
    lin = L.PackedQuantLinear(L.QuantWeight.new_gptq(4, sym, dev[0], None if sym else dev[1], dev[2]))
    y = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
    gemm.packed4_matmul(lin, bf16(x), y)
    w = ((nib.astype(np.int32) - np.repeat(zero, g, 0).astype(np.int32)) * np.repeat(sc.astype(np.float64), g, 0)).T
    got = y.double().cpu().numpy()
    if special:
        same_special(got, x, w)
    block = np.repeat(np.abs(x[rest]).reshape(len(rest), -1, 32).max(-1), 32, -1).astype(np.float64)
    extra = 2.0**-26 * block @ np.abs(w).T if special else 0.0
    assert (np.abs(got[rest] - x[rest].astype(np.float64) @ w.T) <= outlier_bound(x[rest], w) + extra).all()


# ------------------------------------------------------------------------------------------------------- MXFP4 experts, small batches
def experts_layer(experts, hidden, inter, seed, zero_columns=()):
    """A layer and its arrays; in `zero_columns` every other gate and up row of each expert is zero."""
    from oxydllm_b200 import moe
    d = synth.gptoss_moe(experts, hidden, inter, 1, seed=seed)
    d["gu_blocks"] = np.array(d["gu_blocks"])
    gu = d["gu_blocks"].reshape(experts, 2 * inter, hidden // 2)
    for c in zero_columns:
        gu[:, 2::4, c // 2] &= 0xF0 if c % 2 == 0 else 0x0F
        gu[:, 3::4, c // 2] &= 0xF0 if c % 2 == 0 else 0x0F
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


# outliers beside zero weights, infinities and NaN in some rows: stages that come a second time, one stage, several, a last one that is
# short; token blocks with and without them in a CTA's units
@pytest.mark.parametrize("hidden,inter", [(96, 32), (160, 224), (2880, 64), (512, 1600)])
@pytest.mark.parametrize("special", [False, True])
def test_moe_small_batch_outliers_and_infinities(cuda, hidden, inter, special):
    counts = (50, 0, 33, 17)
    x, columns = (special_activations if special else activations_with_outliers)(sum(counts), hidden, seed=hidden)
    if special:
        rest, columns = columns, activations_with_outliers(1, hidden, 0)[1]
    layer, d = experts_layer(len(counts), hidden, inter, seed=hidden + inter, zero_columns=columns)
    ids = np.random.default_rng(1).permutation(np.repeat(np.arange(len(counts)), counts))
    y = layer.forward_experts(bf16(x), torch.from_numpy(ids).cuda())
    layer.check()
    got = y.double().cpu().numpy()
    gb, db = (b.double().cpu().numpy() for b in (layer.gu_bias, layer.dn_bias))
    for e, c in enumerate(counts):
        rows = np.nonzero(ids == e)[0]
        gu = oracle.mxfp4_dequant(d["gu_blocks"][e], d["gu_scales"][e], 2 * inter, hidden).astype(np.float64)
        dn = oracle.mxfp4_dequant(d["dn_blocks"][e], d["dn_scales"][e], hidden, inter).astype(np.float64)
        with np.errstate(invalid="ignore", over="ignore"):
            a = np.stack([(x[r].astype(np.float64) * gu).sum(1) for r in rows]).reshape(len(rows), -1) + gb[e] if c else np.zeros((0, 2 * inter))
            gate, up = np.fmin(a[:, 0::2], 7.0), np.fmin(np.fmax(a[:, 1::2], -7.0), 7.0)  # a NaN takes the limit
            h = (up + 1) * gate / (1 + np.exp(-1.702 * gate))
            ref = h @ dn.T + db[e]
            # gate and up are good to 2^-17 of the sum of |x w|, their product moves by less than 16 times that
            off = 16 * 2.0**-17 * np.minimum(np.abs(x[rows]).astype(np.float64) @ np.abs(gu).T, 1e30).reshape(len(rows), inter, 2).sum(-1)
            bound = 2.0**-8 * (np.abs(h) @ np.abs(dn).T + np.abs(ref)) + off @ np.abs(dn).T + 1e-6
        assert np.array_equal(np.isnan(got[rows]), np.isnan(ref)), e
        ok = np.isfinite(ref) & np.isfinite(bound)
        assert (np.abs(got[rows] - ref)[ok] <= bound[ok]).all(), (e, c)
        if not special:
            assert ok.all()


# more than 44 rows an expert on average: weights unpacked into tensor memory by four teams in turn, accumulators round a ring of columns;
# blocks of up to 192 rows (96, 160 and 300 rows an expert) and of up to 256, whole and beside smaller ones (201 and 218 rows); fewer
# stages of 64 columns than teams, a last stage half past k, more units than SMs, so that blocks of all sizes follow one another in a CTA
@pytest.mark.parametrize("hidden,inter", [(32, 96), (96, 32), (224, 544), (2880, 64), (128, 9600)])
@pytest.mark.parametrize("counts", [(192, 193, 0, 1), (385, 64, 191, 0), (300, 260, 340, 300), (256, 225, 193, 130), (400, 209, 16, 250)])
def test_moe_large_batch_matches_64_bit_experts(cuda, hidden, inter, counts):
    test_moe_small_batch_matches_64_bit_experts(cuda, hidden, inter, counts)


@pytest.mark.parametrize("lo,hi", [(2, 4), (7, 8), (0, 5)])
def test_moe_small_batch_of_a_part_of_the_experts(cuda, lo, hi):
    """Rows per expert decide which kernel serves a call, not how many of the experts are local: with one expert a token, a rank with a part
    of them gives the bits of the whole layer for its tokens, and zeros for the others."""
    layer, _ = experts_layer(8, 256, 512, seed=9)
    layer.top_k = 1
    x = bf16(synth.activations(320, 256, seed=9))
    ids = torch.from_numpy(np.random.default_rng(9).integers(0, 8, 320)).cuda()
    logits = torch.nn.functional.one_hot(ids, 8).float()
    whole, part = layer.forward_with_logits(x, logits), layer.forward_with_logits(x, logits, (lo, hi))
    layer.check()
    local = (ids >= lo) & (ids < hi)
    assert torch.equal(part[local], whole[local]) and not part[~local].any()


def test_moe_small_batch_kernel_survives_weights_that_never_come(cuda):
    ws = torch.zeros(1 << 20, dtype=torch.uint8, device="cuda")
    _lib.call("oxq_selftest_moe_mx_wait_expiry", ws.data_ptr(), ws.numel(), None)
    with pytest.raises(_lib.OxqError, match=r"bounded wait 6[1-7] "):
        gemm.check(ws)
    gemm.check(ws)  # reported once
    test_moe_small_batch_matches_64_bit_experts(cuda, 256, 512, (16, 17, 48, 49))

