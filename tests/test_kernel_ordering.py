"""Orderings inside the tcgen05 kernels that no run shows to be missing: read in the source.  What one thread writes and
another reads needs a barrier between them that orders memory.  The checks are of the text as it stands: they show that a line that
was found missing once is there, not that the order is right, and a rename has to be followed here."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pim-dl-asplos_b200", "csrc")


def _source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


@pytest.mark.parametrize("name,epilogues", [("lut_sparse_umma.cu", 2), ("lut_onehot_umma.cu", 2)])
def test_epilogue_warps_meet_before_they_read(name, epilogues):
    """The lanes of an epilogue warp stage a tile's bias values for one another, and lane 0 alone waits for the
    accumulator: __shfl_sync, which tells the others, orders no memory."""
    waits = list(re.finditer(r"w_ok = [^;]*mbar_wait<256>\(acc_full0", _source(name)))
    assert len(waits) == epilogues
    for w in waits:
        after = _source(name)[w.end():]
        until = after[:after.index("tmem_ld_32x32b_x32(")]
        assert "__syncwarp();" in until[until.index("__shfl_sync("):]


@pytest.mark.parametrize("name", ["lut_sparse_umma.cu", "lut_onehot_umma.cu"])
def test_issuing_warps_take_turns(name):
    """Several warps issue MMAs into one accumulator.  Read-modify-writes of an accumulator are ordered between the
    instructions of one thread; between threads it takes a fence, a barrier and a fence: before its first instruction of a
    slab a warp waits for its turn, behind the last one it hands over."""
    src = _source(name)
    if int(re.search(r"\bkMmaWarps = (\d+)", src).group(1)) == 1:
        return
    for issue in re.finditer(r"if \(elect_one\(\)\) \{\s*const uint32_t b_lo", src):
        before = src[src.rindex("for (uint32_t i = ", 0, issue.start()):issue.start()]
        assert re.search(r"mbar_wait\(turn0 .*tc_fence_after_sync\(\);", before, re.S)
        after = src[issue.start():src.index("umma_commit", issue.start())]
        assert re.search(r"umma_i8.*tc_fence_before_sync\(\);\s*mbar_arrive\(turn0 ", after, re.S)
        break
    else:
        pytest.fail("no issue loop found")


@pytest.mark.parametrize("name,poll,release", [("lut_sparse_umma.cu", "go = *reinterpret_cast<volatile uint32_t*>(ctr) >= p.split;", "mbar_arrive(sums_bar"),
                                               ("lut_onehot_umma.cu", "*reinterpret_cast<volatile uint32_t*>(ctr) >= p.split", "s_misc[2] = go;")])
def test_split_sums_are_read_behind_a_fence(name, poll, release):
    """The thread that sees all slices of a tile stored releases the others, and they read what the counter stands for: the
    fence belongs to that thread, before the release."""
    src = _source(name)
    seen = src.index(poll)
    assert "__threadfence();" in src[seen:src.index(release, seen)]


def test_the_polling_warp_meets_behind_the_fence():
    src = _source("lut_sparse_umma.cu")
    told = src.index("__shfl_sync(0xffffffffu, go, 0);")
    assert "__syncwarp();" in src[told:src.index("} else {", told)]


def test_the_search_hands_its_columns_over_in_order():
    """The warp that reads last has the next columns computed into those all four have read: its lanes' reads, and what they
    wrote for the next tile, are ordered before the count by lane 0, and the count before the instructions of whichever lane
    issues them.  The kernel that wants all tensor memory is let in behind the allocation."""
    src = _source("ccs_umma.cu")
    release = src[src.index("auto release = "):src.index("auto settle_all = ")]
    assert re.search(r"tc_fence_before_sync\(\);\s*__syncwarp\(\);.*atom\.acq_rel\.cta.*__shfl_sync\(.*__syncwarp\(\);.*issue\(", release, re.S)
    issue = src[src.index("auto issue = "):src.index("auto release = ")]
    assert issue.index("tc_fence_after_sync();") < issue.index("elect_one()")
    convert = src[src.index("auto convert = "):src.index("auto issue = ")]
    assert convert.rstrip().endswith("fence_proxy_async_smem();\n    };")
    kernel = src[src.index("ccs_umma_kernel("):]
    assert kernel.index("tmem_alloc(") < kernel.index("__syncthreads();") < kernel.index("pdl_launch_dependents();")


def test_the_searching_warps_leave_together():
    """Full-mask instructions follow each wait of the search, so its answer is one for the warp, and a warp whose wait has
    run out does nothing more; the columns are handed back when what is in flight has had time to end."""
    src = _source("ccs_umma.cu")
    assert not re.search(r"\bmbar_(try_)?wait(_limited)?\b", src)
    waits = list(re.finditer(r"mbar_wait_warp\([^;]*;", src))
    assert waits
    for w in waits:
        assert re.match(r"\s*if \(!ok\) break;", src[w.end():])
    down = src[src.rindex("__syncthreads();", 0, src.index("tmem_dealloc(")) - 400:src.index("tmem_dealloc(")]
    assert down.index("if (s_abort)") < down.index("clock64()") < down.index("report_error(")


@pytest.mark.parametrize("name", ["lut_sparse_umma.cu", "lut_onehot_umma.cu"])
def test_no_lane_leaves_a_warp_alone(name):
    """Waits of whole warps: between one whose answer is a lane's own and the vote on it no lane takes another way."""
    src = _source(name)
    own = list(re.finditer(r"\bok = (ok && )?mbar_wait\(", src))
    assert len(own) >= 3
    for w in own:
        behind = src[w.end():]
        assert not re.search(r"\b(break|continue|return)\b", behind[:behind.index("__all_sync(0xFFFFFFFFu, ok)")])
    assert len(re.findall(r"__all_sync\(0xFFFFFFFFu, ok\)", src)) == 2
