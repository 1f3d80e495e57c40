"""Kernels that are launched before the one ahead of them on the stream has finished: what may stand in front of
``pdl_wait()``, checked on the sources (a violation is a race, which no run shows reliably)."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oxydllm_b200", "csrc")
WAIT = re.compile(r"\bpdl_wait(_zero)?\(\)")
# The GEMVs that include/oxq.h names: their weights, scales and zero points may be read early and through the read-only path.
READ_WEIGHTS_EARLY = {"awq_gemv_group_kernel", "awq_gemv_tma_kernel", "fp8_gemv_kernel", "mxfp4_gemv_kernel", "q40_gemv_kernel",
                      "q4k_gemv_kernel", "q6k_gemv_kernel", "q6k_gemv_wide_kernel", "q80_gemv_kernel"}
# Launched behind a kernel that triggers only after its own wait: whatever may write weights has finished before these start.
BEHIND_A_SPLIT = {"packed_mx_tc_kernel": "packed_mx_split_kernel", "moe_mx_kernel": "moe_mx_split_kernel"}


def early_kernels(paths=None):
    """Name -> (signature, body), without comments, of every ``__global__`` function that waits for the kernel ahead."""
    found = {}
    for path in paths or sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\(.*?\)\s+)?(\w+)\s*\(([^;{]*)\)\s*\{", text, re.S):
            body = text[m.end():text.index("\n}\n", m.end())]
            if WAIT.search(body):
                found[m.group(1)] = (m.group(2), body)
    return found


def reads_weights_out_of_order(signature, body):
    """What lets a load of this kernel be served, or be moved, ahead of the kernel that wrote the data."""
    return re.findall(r"const\s+\w+\s*\*\s*__restrict__\s*\w+", signature) + re.findall(r"__ldg\(", body)


def test_the_kernels_are_found():
    """Every kernel that can be launched early is looked at: each launch that sets the attribute names one of them."""
    names = set(early_kernels())
    assert READ_WEIGHTS_EARLY | set(BEHIND_A_SPLIT) | set(BEHIND_A_SPLIT.values()) <= names
    assert {"packed_group_tc_kernel", "awq_fused_tc_kernel", "gated_act_rows_kernel", "gemm_bf16_tn_kernel", "gemm_bf16_tn_2cta_kernel",
            "moe_route_kernel", "moe_dispatch_small_kernel", "moe_combine_kernel", "awq_slab16_bf16_kernel", "fp8_slab16_bf16_kernel",
            "q4k_slab_bf16_kernel", "q80_slab_bf16_kernel", "q40_slab_bf16_kernel", "q6k_slab_bf16_kernel", "gptq4_slab_bf16_kernel",
            "gptq_gemv_kernel", "w8a16_gemv_kernel", "gptq4_gemv_mma_kernel"} <= names
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for name in re.findall(r"launch_early\((\w+)", text):
            assert name in names or name == "void", (path, name)


@pytest.mark.parametrize("name", sorted(set(early_kernels()) - READ_WEIGHTS_EARLY - set(BEHIND_A_SPLIT)))
def test_weights_come_in_the_order_of_the_stream(name):
    """Callers of all entry points but those GEMVs may write weights with the kernel just ahead: nothing is loaded before the wait, and
    nothing through the read-only path, which may be served before it."""
    signature, body = early_kernels()[name]
    before = body[:WAIT.search(body).start()]
    assert not re.search(r"tma_load|bulk_copy|__ldc?[gsa]\(|ld_produced|ld_ordered|load_as_f32|ld\.global|\bp\.(qzeros|scales|bias|x|y)\b", before)
    assert reads_weights_out_of_order(signature, body) == []


@pytest.mark.parametrize("line", ["void k(const uint8_t *__restrict__ w)", "void k(const uint8_t *w)"])
def test_the_rule_sees_signatures_and_bodies(line, tmp_path):
    src = tmp_path / "k.cu"
    src.write_text("__global__ void __launch_bounds__(256)\n%s\n{\n    pdl_wait();\n    y[0] = %s;\n}\n"
                   % (line[5:], "w[0]" if "restrict" in line else "__ldg(w)"))
    assert reads_weights_out_of_order(*early_kernels([str(src)])["k"])


@pytest.mark.parametrize("name", sorted(BEHIND_A_SPLIT.values()))
def test_split_kernels_trigger_after_their_own_wait(name):
    body = early_kernels()[name][1]
    assert WAIT.search(body).start() < body.index("pdl_launch_dependents()")


def test_block_scaled_kernel_loads_only_weights_before_the_wait():
    """Its weight producer and unpack warps run ahead; each other role waits for the split kernel before its loop."""
    body = early_kernels()["packed_mx_tc_kernel"][1]
    roles = re.split(r"\n    (?:\} else )?if \((?=[^\n]*\bwarp\b)", body)
    for role in roles:
        if re.search(r"&xmap|p\.sf\b|p\.sx\b", role):
            assert WAIT.search(role) and WAIT.search(role).start() < re.search(r"&xmap|p\.sf\b|p\.sx\b", role).start()


@pytest.mark.parametrize("name", sorted(n for n, (_, b) in early_kernels().items() if re.search(r"\b(mbar_wait|mbar_test|mx_wait[23]?)\(", b)
                                        and n != "packed_mx_tc_kernel"))
def test_bounded_waits_do_not_count_the_time_of_the_kernel_ahead(name):
    body = early_kernels()[name][1]
    assert WAIT.search(body).start() < re.search(r"\b(mbar_wait|mbar_test|mx_wait[23]?)\(", body).start()


def test_what_a_kernel_ahead_writes_is_not_read_through_the_read_only_path():
    """``__ldg`` may be served before ``pdl_wait``: in the GEMVs for weights, scales and zero points only."""
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        if WAIT.search(text):
            assert not re.search(r"__ldg\([^;]*?\b(src|xin|p\.x|p\.gu|gu|pair_expert)\b", text), path
