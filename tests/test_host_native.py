"""The native host side of decode calls: what it takes it does as the Python code does, and what it does not take is left to that."""
import numpy as np
import pytest
import torch
from torch.utils.flop_counter import FlopCounterMode

from oxydllm_b200 import _lib, formats as F, gemm, linear as L, synth


def test_leaves_what_is_not_a_plain_cuda_tensor(tmp_path):
    host = _lib.host()
    x = torch.zeros(2, 256, dtype=torch.bfloat16)
    for args in ((), (1,) * 8, (x, x, None, F.GGML_Q4_0, 256, 64, 2, 32), (None, x, None, "type", 256, 64, 2, 32)):
        assert host.gguf(*args) is None
    assert host.packed4(x, x, x, x, None, 256, 64, 128, 4, False, False, (8, 8)) is None
    assert host.ffn(x, x, x, x, 256, 64, 128, 1) is None and host.fp8(x, x, x, None, 256, 64, 16) is None
    with pytest.raises(TypeError):
        host.keep(0, "tensor")
    with pytest.raises(ValueError):
        host.keep(0, x)


def _layers():
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    words = lambda a: dev(a.view(np.int32))  # noqa: E731
    qw, qz, sc = synth.awq_layer(512, 256, 128, seed=1)
    awq = L.PackedQuantLinear(L.QuantWeight.new_awq(4, words(qw), words(qz), dev(sc)))
    odd = L.PackedQuantLinear(L.QuantWeight.new_awq(4, words(qw[:, :25].copy()), words(qz[:, :25].copy()), dev(sc[:, :200].copy())))
    gq = torch.randint(-2**31, 2**31 - 1, (64, 256), dtype=torch.int32, device="cuda")
    gptq = L.PackedQuantLinear(L.QuantWeight.new_gptq(4, True, gq, None, dev(sc)), torch.ones(256, dtype=torch.bfloat16, device="cuda"))
    q4 = L.QLinear(F.GGML_Q4_0, dev(synth.gguf_layer(F.GGML_Q4_0, 256, 512, seed=2)), 256, 512, torch.ones(256, device="cuda"))
    q4f = L.QLinear(F.GGML_Q4_K, dev(synth.gguf_layer(F.GGML_Q4_K, 256, 512, seed=2)), 256, 512, out_dtype=torch.float32)
    w, s = synth.fp8_layer(256, 512, seed=3)
    return [awq, odd, gptq, L.GatedFfnProjection(awq, "silu"), q4, q4f, L.Fp8Linear(dev(w).view(torch.uint8).view(torch.float8_e4m3fn), dev(s)),
            L.Fp8Linear(dev(w).view(torch.uint8).view(torch.float8_e4m3fn))]


@pytest.mark.gpu
@pytest.mark.parametrize("m", [1, 3, 8, 9, 16, 33, 70, 300])
def test_same_results_as_the_python_code(cuda, m, monkeypatch):
    """Batches on both sides of the choices, x of two and three dimensions, on 16 and 8 bytes, and strided."""
    flat = torch.from_numpy(synth.activations(2 * m, 512, seed=m)).to(torch.bfloat16).cuda()
    off = torch.empty(m * 512 + 4, dtype=torch.bfloat16, device="cuda")[4:].view(m, 512).copy_(flat[:m])
    for lin in _layers():
        for x in (flat[:m], flat.view(2, m, 512), flat[:m].view(1, m, 512), off, flat[::2]):
            try:
                with monkeypatch.context() as p:
                    p.setattr(gemm, "native", lambda: None)
                    want = lin.forward(x)
            except _lib.OxqError as e:  # a call that is refused stays refused
                with pytest.raises(_lib.OxqError, match=str(e.status)):
                    lin.forward(x)
                continue
            got = lin.forward(x)
            assert got.shape == want.shape and got.dtype == want.dtype and got.is_contiguous() and torch.equal(got, want)


@pytest.mark.gpu
def test_takes_plain_calls_and_no_others(cuda):
    lin = _layers()[4]
    x = torch.from_numpy(synth.activations(2, 512, seed=1)).to(torch.bfloat16).cuda()
    want = lin.forward(x)  # (the first call makes the flag words)
    host = gemm.native()
    call = lambda x: host.gguf(x, lin.blocks, lin.bias, lin.ggml_type, 512, 256, _lib.OXQ_BF16, 32)  # noqa: E731
    assert torch.equal(call(x), want)
    for bad in (x.float(), x[:, :256], x[0], x.t().contiguous().t(), x[:0], x.cpu(), x.to_sparse()):
        assert call(bad) is None
    assert torch.func.vmap(lambda r: torch.zeros(1) if call(r) is None else 1 / 0)(x[None]).shape == (1, 1)
    with FlopCounterMode(display=False):
        assert call(x) is None
    with torch.inference_mode():
        assert call(x).is_inference()
    with pytest.raises(ValueError):
        lin.forward(x[:, :256])
