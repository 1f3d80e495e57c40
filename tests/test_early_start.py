"""Kernels that are launched before the one ahead of them on the stream has finished: what may stand in front of
``pdl_wait()``, checked on the sources (a violation is a race, which no run shows reliably)."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oxydllm_b200", "csrc")


def kernels():
    """Name -> body, without comments, of every ``__global__`` function that calls ``pdl_wait``."""
    found = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__[^;{]*?(\w+)\s*\(const[^{;]*\)\s*\{", text):
            body = text[m.end():text.index("\n}\n", m.end())]
            if "pdl_wait()" in body:
                found[m.group(1)] = body
    return found


def test_the_kernels_are_found():
    assert {"packed_group_tc_kernel", "q6k_gemv_wide_kernel", "awq_gemv_tma_kernel", "gated_act_rows_kernel"} <= set(kernels())


def test_grouped_kernel_reads_nothing_before_the_wait():
    """Its callers were ordered by the stream before it started early: weights may come from the kernel just ahead."""
    before = kernels()["packed_group_tc_kernel"].split("pdl_wait()")[0]
    assert not re.search(r"tma_load|bulk_copy|__ldg|__ldcg|ld\.global|p\.(qzeros|scales|bias|y)\b", before)


@pytest.mark.parametrize("name", ["packed_group_tc_kernel", "awq_gemv_tma_kernel", "q6k_gemv_wide_kernel"])
def test_bounded_waits_do_not_count_the_time_of_the_kernel_ahead(name):
    body = kernels()[name]
    assert body.index("pdl_wait()") < re.search(r"\b(mbar_wait|gt_wait|mbar_test)\w*\(", body).start()


def test_what_a_kernel_ahead_writes_is_not_read_through_the_read_only_path():
    """``__ldg`` and ``const __restrict__`` may be served before ``pdl_wait``: for weights, scales and zero points only."""
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        if "pdl_wait()" in text:
            assert not re.search(r"__ldg\([^;]*?\b(src|xin|p\.x|p\.gu|gu|pair_expert)\b", text), path
    for name, body in kernels().items():
        assert not re.search(r"const\s+\w+\s*\*\s*__restrict__", body.split("{")[0]), name
