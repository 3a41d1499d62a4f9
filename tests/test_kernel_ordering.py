"""Orderings inside the tcgen05 kernels that no run shows to be missing: read in the source.  What one thread writes and
another reads needs a barrier between them that orders memory."""
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
