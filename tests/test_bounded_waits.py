"""What the tensor-core kernels do once a bounded wait has run out, read from their sources: a wait is never made to run out on a GPU,
because what it guards against (copies that land in memory of another block, an aligned instruction that half a warp executes, an
accumulator that lacks products) is not an error that a GPU reports."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llama.cu_b200", "csrc")
FILES = ["gemm_tc.cu", "gemm_pair.cu", "attention_tc.cu", "latent_tc.cu"]


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def kernels(text):
    """The bodies of the kernels that own tensor memory."""
    return [b for b in re.split(r"\n__global__ ", text)[1:] if "tcgen05.alloc" in b]


@pytest.mark.parametrize("name", FILES)
def test_a_warp_loads_an_accumulator_as_a_whole(name):
    for body in kernels(source(name)):
        for load in re.finditer(r"tc_ld16\(|at_ld32\(", body):
            wait = body.rfind("tc_mbar_wait(", 0, load.start())
            if wait >= 0:  # the decision that follows the wait is one of the whole warp (or of all four warps)
                line = body.rfind("\n", 0, wait)
                assert re.search(r"__all_sync|lt_sync_and", body[line:load.start()]), body[line:load.start()][:200]


@pytest.mark.parametrize("name", ["gemm_tc.cu", "gemm_pair.cu"])
def test_an_accumulator_that_lacks_products_is_not_handed_over(name):
    for body in kernels(source(name)):
        commits = list(re.finditer(r"commit\w*\(tc_smem\(&sh->tmem_full", body))
        assert commits
        for c in commits:
            before = body[:c.start()].rstrip().split("\n")
            assert re.search(r"if \(!?stop\)|abort_flag", before[-1] + before[-2]), before[-2:]


@pytest.mark.parametrize("name", FILES)
def test_a_block_leaves_after_its_copies_and_products(name):
    text = source(name)
    drains = re.search(r"tc_leave\(TcShared.*?\n}\n", text, re.S)
    for body in kernels(text):
        if name == "latent_tc.cu":  # its producer waits for its own ring
            assert "never" in body
            continue
        leave = body[body.rfind("tcgen05.fence::before_thread_sync"):body.rfind("tcgen05.dealloc")]
        if "tc_leave(sh, warp, issued, n_stages)" in leave:
            leave += drains.group(0)
        assert "abort_flag" in leave and "tc_warp_drain_ring(" in leave and re.search(r"commit\w*\(tc_smem\(&sh->drain\)", leave), leave
        assert leave.index("__syncthreads") < leave.index("abort_flag") or "tc_leave" in leave  # when no warp can give up any more
        assert len(re.findall(r"\+\+\w*issued|issued = ", body)) >= 2
