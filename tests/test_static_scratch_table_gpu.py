"""lutamm_amm_static_scratch at shapes where it contracts on the tensor cores.  A 16-byte aligned table is contracted as it is:
every centroid count, both tile widths, column counts whose rows straddle sectors, half-filled last slabs and tiles.  Any
other is laid out first: in one piece, in several pieces of columns (also with a ragged last one), and with the indices
taking most of the array."""
import ctypes

import numpy as np
import pytest

import oracle
import pim_dl_asplos_b200 as P
from pim_dl_asplos_b200 import synth

pytestmark = pytest.mark.gpu


PIECES = [(300, 256, 512, 2, 16), (520, 768, 1616, 2, 16), (1100, 512, 3088, 4, 64), (2300, 2048, 1040, 2, 8), (9, 1024, 2064, 4, 16)]
WHOLE = [(1300, 512, 144, 2, 8), (1500, 768, 272, 2, 32), (512, 768, 1072, 4, 64), (385, 1024, 2064, 4, 128), (385, 512, 4160, 2, 256),
         (3000, 832, 2064, 4, 16), (257, 768, 3104, 4, 64)]


@pytest.mark.parametrize("M,K,N,v,CT,offset", [c + (o,) for o in (0, 4) for c in PIECES] + [c + (0,) for c in WHOLE])   # offset of the table from a 16-byte boundary
def test_static_scratch_against_the_oracle(M, K, N, v, CT, offset):
    import torch
    c = synth.make_case(M=M, K=K, N=N, v=v, CT=CT, seed=M)
    x, cen, bias = (torch.from_numpy(a).cuda() for a in (c.x, c.centroid, c.bias))
    lut = torch.empty(c.lut.size + 16, dtype=torch.int8, device="cuda")[offset:offset + c.lut.size]
    lut.copy_(torch.from_numpy(c.lut).flatten())
    y = torch.full((M, N), float("nan"), device="cuda")
    torch.cuda.synchronize()
    ip, lp = P.make_params(M, K, N, K // v, CT, c.scale, c.lut_bias)
    lib = P.load_library()
    for _ in range(2):
        rc = lib.lutamm_amm_static_scratch(0, None, x.data_ptr(), cen.data_ptr(), lut.data_ptr(), bias.data_ptr(), y.data_ptr(),
                                           ctypes.byref(ip), ctypes.byref(lp))
        assert rc == P.OK, lib.lutamm_static_scratch_last_error().decode()
    want = oracle.amm(c.x, c.centroid, c.lut, c.bias, c.scale, c.lut_bias)[0]
    assert np.array_equal(y.cpu().numpy().view(np.uint32), want.view(np.uint32))
