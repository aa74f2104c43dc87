"""What a kernel reads before it has waited for the kernel ahead of it.  Read from the sources: what an early read returns is a matter
of time on a GPU, and none is made to happen there."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tensorwarp_b200", "csrc")
READS = r"tma_load_\w+\(|bulk_g2s\(|__ldg\(|reinterpret_cast<const (?:float4|uint4|uint2|__half2)\*>"


def kernels(name):
    """(name, body) of the kernels of a file, without comments."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    parts = re.split(r"__global__ void __launch_bounds__\([^\n]*\n", text)[1:]
    return [(re.match(r"\s*(\w+)\(", p).group(1), p) for p in parts]


# kernels of calls that may leave TWM_FLAG_PDL clear: (file, how many)
WAIT_FIRST = {"twm_gemv_simt.cuh": 1, "twm_gemv_mma.cuh": 3, "twm_gemm_tc.cuh": 2, "twm_gemm_tcw.cuh": 1, "twm_gemm_tcr.cuh": 1}


@pytest.mark.parametrize("name", WAIT_FIRST)
def test_kernels_of_plain_calls_wait_before_they_read(name):
    """A call without the flag is launched beside the kernel before; each of its kernels, the product behind a pre-pass too, waits in every
    thread before anything is read."""
    found = kernels(name)
    assert len(found) == WAIT_FIRST[name]
    for kernel, body in found:
        at = re.search(r"pdl_begin\((?:p\.)?wait_first\);", body)
        assert at and "pdl_launch_dependents" not in body, kernel
        first = re.search(READS, body)
        assert first is None or at.start() < first.start(), kernel
        # reached by every thread: outside any block but the kernel's own
        assert body[:at.start()].count("{") - body[:at.start()].count("}") == 1, kernel


@pytest.mark.parametrize("name,kernel", [("twm_decode_ops.cuh", "rmsnorm_kernel"), ("twm_decode_ops.cuh", "attn_chunk_kernel")])
def test_factors_and_biases_are_read_after_the_wait(name, kernel):
    """With TWM_FLAG_PDL too: what the kernel before may write is no more than asked for towards L2 ahead of the wait."""
    body = dict(kernels(name))[kernel]
    ahead = body[:body.index("pdl_wait_prior_grids();")]
    assert "l2_prefetch(" in ahead and not re.search(READS + r"|\b(?:gamma|bias)\[", ahead)
