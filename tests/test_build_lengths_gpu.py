"""The table's construction at the sub-vector lengths of the hidden-size sweep (2560 / 256, 5120 / 256 and 32), whose weights
stay in registers: one column group, a ragged block of columns, more centroids than are summed together.  Bytes are equal."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("v", [10, 20, 32])
@pytest.mark.parametrize("CB,CT,N", [(1, 1, 4), (3, 16, 1028), (2, 9, 1020), (5, 33, 260)])
def test_bytes_equal_the_stated_order(ctx, v, CB, CT, N):
    rng = np.random.default_rng(v * 100 + CT)
    cen = rng.standard_normal((CB, CT, v), dtype=np.float32)
    w = (rng.standard_normal((CB * v, N)) * 0.02).astype(np.float32)
    w[:, ::7] = 0
    want, scale, bias = oracle.build_lut(cen, w)
    got, got_scale, got_bias = ctx.build_lut(cen, w)
    assert np.array_equal(got, want) and np.float32(got_scale) == np.float32(scale) and got_bias == bias
