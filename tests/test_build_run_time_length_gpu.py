"""Table construction at sub-vector lengths that have no instance of their own: centroids eight at a time, the last group
partly filled, columns past the last block."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("CB,v,CT,N", [(5, 3, 1, 16), (4, 10, 7, 1040), (3, 20, 8, 48), (2, 32, 9, 2064), (7, 5, 16, 1024), (2, 6, 255, 32)])
def test_against_the_oracle(ctx, CB, v, CT, N):
    rng = np.random.default_rng(CB + CT + N)
    cen = rng.standard_normal((CB, CT, v), dtype=np.float32)
    weight = rng.standard_normal((CB * v, N), dtype=np.float32)
    got = ctx.build_lut(cen, weight)
    want = oracle.build_lut(cen, weight)
    assert np.array_equal(np.asarray(got[0]), np.asarray(want[0]))
    assert got[1] == want[1]
