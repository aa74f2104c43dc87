"""CTAs of a cluster that add up one another's sums: no CTA stores C when a wait of any of them ran out.  Read from the sources: a wait
that runs out leaves copies in flight, so none is made to on a GPU."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tensorwarp_b200", "csrc")
FILES = {"twm_gemv_simt.cuh": 1, "twm_gemv_mma.cuh": 2, "twm_gemm_tcw.cuh": 1, "twm_gemm_tcr.cuh": 1, "twm_dense_tcs.cuh": 1, "twm_dense_f32tc.cuh": 1}
SUMS = r"cluster_sum4\w*\(|slice_sum_store<"


def kernels(name):
    """Bodies of the kernels of a file that read sums of other CTAs or push sums to them, without comments."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    return [b for b in text.split("__global__")[1:] if re.search(SUMS + r"|st_cluster_f32\(", b)]


@pytest.mark.parametrize("name", FILES)
def test_no_cta_of_a_cluster_stores_after_an_expired_wait(name):
    found = kernels(name)
    assert len(found) == FILES[name]
    for body in found:
        for use in re.finditer(SUMS, body):
            if use.group() == "cluster_sum4_met(":                     # the flags of all CTAs come with the sums; the store hangs on them
                assert re.match(r"cluster_sum4_met\([^;]*\)\) store_c4\(", body[use.start():]) and "if (" in body[use.start() - 40:use.start()]
                continue
            # every thread has announced itself and met the others, and what that returned guards the statement
            assert body.count("cluster_started();") == 1
            meet = body.index("cluster_meet(abort_flag)")
            assert meet < use.start()
            assert re.search(r"if \(cluster_meet\(abort_flag\)\)|if \(all_ok\)|&& all_ok|if \(!all_ok\)", body[max(0, meet - 40):use.start()])
        for push in re.finditer(r"st_cluster_f32\(", body):          # partial sums pushed to a leader, which looks at its own flag
            told, tail = body[:push.start()].rindex("cluster_tell_abort(abort_flag)"), body[push.start():]
            assert body.index("cluster_started();") < body[:told].rindex("cluster_wait_started();") and "cluster_sync_all()" not in body[told:push.start()]
            assert tail.index("cluster_sync_all()") < tail.index("*abort_flag == 0")


def test_every_warp_reaches_the_barriers_of_its_cluster():
    """Producer and other warps that hold no sums: as many barriers as those that do."""
    for name in ("twm_gemm_tcw.cuh", "twm_gemm_tcr.cuh"):
        assert kernels(name)[0].count("cluster_meet(abort_flag)") == 2
    for name, body in (("twm_gemv_simt.cuh", kernels("twm_gemv_simt.cuh")[0]), ("twm_gemv_mma.cuh", kernels("twm_gemv_mma.cuh")[1])):
        assert body.count("cluster_sync_all()") == 4 and "{ cluster_sync_all(); cluster_sync_all(); }" in body, name
