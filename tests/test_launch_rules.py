"""What a call launches, by size, type and alignment: the library's objects on a runtime that only logs (fake_cudart.cpp)."""
import ctypes
import glob
import os
import shutil
import subprocess

import pytest

import pim_dl_asplos_b200 as P

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "pim-dl-asplos_b200", "csrc")
OBJECTS = sorted(glob.glob(os.path.join(CSRC, "build", "*.o")))
INCLUDE = "/usr/local/cuda/include"

pytestmark = pytest.mark.skipif(not (OBJECTS and shutil.which("g++") and os.path.exists(os.path.join(INCLUDE, "cuda_runtime.h"))),
                                reason="the library's objects or the toolkit's headers are not here")


class _Library:
    def __init__(self, path):
        self.lib = ctypes.CDLL(path)
        self.lib.fake_log.restype = ctypes.c_char_p
        self.ctx = ctypes.c_void_p()
        assert self.lib.lutamm_create(ctypes.byref(self.ctx), 0) == P.OK
        self.memory = ctypes.create_string_buffer(1 << 26)   # stands for any buffer of the caller: nothing is run on it
        self.base = (ctypes.addressof(self.memory) + 255) // 256 * 256

    def log(self):
        return self.lib.fake_log().decode().splitlines()

    def amm(self, M, K, N, v=2, CT=16, plan=None):
        """Launches of lutamm_amm on device buffers."""
        at, L = ctypes.c_void_p(self.base), self.lib
        ip, lp = P.make_params(M, K, N, K // v, CT, 0.01)
        assert L.lutamm_load_weights(self.ctx, 0, at, at, at, ctypes.byref(ip), ctypes.byref(lp)) == P.OK
        if plan:
            assert L.lutamm_set_plan(self.ctx, 0, ctypes.byref(P.Plan(**plan))) == P.OK
        for _ in range(2):   # the first call lays the table out
            self.log()
            assert L.lutamm_amm(self.ctx, 0, at, at, ctypes.c_uint32(M), ctypes.c_uint32(P.FLAG_ASYNC)) == P.OK
        return self.log()


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    path = str(tmp_path_factory.mktemp("fake") / "libfake.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", CSRC, "-I", INCLUDE, "-o", path,
                    os.path.join(HERE, "fake_cudart.cpp")] + OBJECTS + ["-ldl"], check=True, timeout=300)
    return _Library(path)


@pytest.mark.parametrize("early,M,K,N,v,CT", [
    (1, 128, 768, 2304, 2, 16), (1, 256, 768, 3072, 2, 16), (1, 64, 1280, 3840, 4, 16), (1, 128, 768, 2304, 2, 32), (1, 128, 768, 2304, 4, 8),
    (0, 512, 768, 3072, 2, 16),       # more than four search CTAs per idle SM
    (0, 320, 768, 2304, 2, 16),       # four idle SMs
    (0, 320, 768, 3072, 4, 64), (0, 192, 2560, 7680, 10, 16), (0, 256, 768, 3072, 8, 16),   # no light search
    (0, 48, 1024, 3072, 4, 16),       # the next call may gather rows
    (0, 12608, 768, 3072, 2, 16)])    # several tiles per pair
def test_who_launches_the_next_kernel_early(fake, early, M, K, N, v, CT):
    contraction = [ln for ln in fake.amm(M, K, N, v, CT) if "lut_sparse_kernel" in ln]
    assert len(contraction) == 1 and contraction[0].endswith(f"early={early}")


def _rows_bytes(M, K, N, CT):
    return M * ((N + 127) // 128) * K * CT * 4   # centroids read by all CTAs


@pytest.mark.parametrize("launches,M,K,N,v,CT", [
    (1, 1, 768, 768, 2, 16), (1, 20, 768, 768, 2, 16), (2, 24, 768, 768, 2, 16), (2, 4, 1024, 4096, 2, 16),   # 6.5 MB: the search alone has a short form
    (1, 12, 768, 2304, 8, 16), (2, 48, 768, 768, 8, 16),                                                      # 13 MB: with 128 floats a codebook
    (1, 24, 768, 768, 4, 13), (1, 12, 768, 768, 2, 64), (2, 4, 1024, 4096, 4, 32),                            # 16 MB: it has none
    (2, 4, 768, 768, 2, 13), (2, 4, 780, 768, 10, 16)])                                                     # no such instance
def test_who_searches_in_the_row_gather(fake, launches, M, K, N, v, CT):
    log = fake.amm(M, K, N, v, CT)
    assert len(log) == launches and "lut_rows_kernel" in log[-1]
    if launches == 1:
        assert _rows_bytes(M, K, N, CT) <= 16e6


def _static(fake, M, K, N, v, CT, offset=0):
    at, lib = ctypes.c_void_p(fake.base), fake.lib
    ip, lp = P.make_params(M, K, N, K // v, CT, 0.01)
    fake.log()
    rc = lib.lutamm_amm_static_scratch(0, None, at, at, ctypes.c_void_p(fake.base + offset), at, at, ctypes.byref(ip), ctypes.byref(lp))
    assert rc == P.OK
    return fake.log()


@pytest.mark.parametrize("form,M,K,N,v,CT", [
    ("rows", 1, 768, 3072, 2, 16), ("rows", 64, 768, 768, 4, 16), ("rows", 29, 1408, 12464, 4, 128), ("rows", 252, 896, 224, 8, 8),
    ("table", 256, 768, 3072, 2, 16), ("table", 1024, 768, 2304, 4, 64), ("table", 512, 768, 3072, 4, 32), ("table", 256, 4096, 4096, 8, 16),
    ("table", 256, 768, 2304, 4, 64), ("table", 128, 768, 3072, 4, 32), ("table", 256, 3072, 768, 2, 16),
    ("gather", 122, 160, 15440, 10, 16), ("gather", 64, 32, 8192, 2, 13), ("gather", 66000, 16, 16, 2, 200)])
def test_how_the_static_call_contracts(fake, form, M, K, N, v, CT):
    """The fastest by measurement of all three at these sizes, and no split of the codebook axis, for which it has no scratch."""
    log = _static(fake, M, K, N, v, CT)
    assert len(log) == 2
    assert {"rows": "lut_rows_kernel", "table": "lut_sparse_kernel", "gather": "lut_gather_kernel"}[form] in log[-1]
    assert all("split=1" in ln for ln in log if "lut_sparse_kernel" in ln)


@pytest.mark.parametrize("early,M,K,N,v,CT", [("110", 512, 768, 3072, 2, 16), ("000", 1024, 768, 3072, 2, 16), ("00000", 384, 512, 8192, 2, 16),
                                              ("11110", 640, 512, 8192, 2, 16), ("0", 300, 256, 512, 2, 16)])
def test_who_launches_the_next_pieces_layout_early(fake, early, M, K, N, v, CT):
    """An unaligned table is laid out in pieces.  Up to eight CTAs of the next layout per SM without a tile; nothing behind the last piece."""
    log = [ln for ln in _static(fake, M, K, N, v, CT, offset=4) if "lut_sparse_kernel" in ln]
    assert "".join(ln[-1] for ln in log) == early


@pytest.mark.parametrize("tile,M,K,N,v,CT", [(64, 1300, 512, 144, 2, 8), (64, 1500, 768, 272, 2, 32), (64, 512, 768, 1072, 4, 64), (64, 385, 1024, 2064, 4, 128),
                                             (128, 385, 512, 4160, 2, 256), (128, 3000, 832, 2064, 4, 16), (128, 512, 768, 3072, 2, 16)])
def test_an_aligned_table_is_contracted_as_it_is(fake, tile, M, K, N, v, CT):
    """One launch behind the search, no layout of the table; the tile width by how N lies to the sectors."""
    log = _static(fake, M, K, N, v, CT)
    assert len(log) == 2 and f"lut_sparse_kernelILj{tile}E" in log[1]


def test_an_unaligned_table_is_not_gathered_by_rows(fake):
    assert "lut_rows_kernel" in _static(fake, 1, 768, 768, 2, 16)[-1]
    assert not any("lut_rows_kernel" in ln for ln in _static(fake, 1, 768, 768, 2, 16, offset=4))


@pytest.mark.parametrize("M,K,N,CT,rows", [(600, 1088, 1248, 13, True), (65535, 1024, 128, 200, True), (65536, 1024, 128, 200, False)])
def test_rows_without_a_tensor_core_form(fake, M, K, N, CT, rows):
    """13 and 200 centroids have no contraction; a token is a block of the row gather's grid.z."""
    assert ("lut_rows_kernel" in fake.amm(M, K, N, 2, CT)[-1]) == rows


@pytest.mark.parametrize("shares,M,CB,N", [(2, 600, 4096, 16), (2, 600, 4098, 16), (2, 600, 4610, 32), (8, 2, 17000, 16), (1, 260, 511, 144), (4, 4, 1024, 768), (1, 64, 384, 768)])
def test_shares_of_the_row_gather(fake, shares, M, CB, N):
    """The split of the codebook axis, and the instance for shares of more than 256 codebooks."""
    last = fake.amm(M, 2 * CB, N, 2, 13)[-1]
    assert "lut_rows_kernel" in last and last.split()[-3] == str(shares)
    assert f"Lb{int((CB + shares - 1) // shares > 256)}E" in last


@pytest.mark.parametrize("tensor,M,K,v,CT,offset", [
    (1, 32768, 768, 4, 64, 0), (1, 8192, 768, 4, 64, 0), (0, 8192, 3072, 2, 32, 0), (1, 4096, 3072, 4, 128, 0), (1, 32768, 768, 8, 32, 0),
    (0, 7812, 768, 4, 64, 0), (0, 32768, 768, 2, 16, 0), (0, 32768, 768, 4, 16, 0), (0, 32768, 2560, 10, 32, 0),   # too little to save
    (1, 512, 8192, 4, 128, 0), (0, 390, 10240, 4, 128, 0), (0, 768, 10240, 4, 128, 0),   # waves that few tokens of many codebooks leave empty
    (0, 32768, 768, 4, 64, 4),     # activations that are not 16-byte aligned
    (0, 65536, 8 * 191, 8, 64, 0)])   # codebooks that do not divide among CTAs
def test_who_searches_on_the_tensor_cores(fake, tensor, M, K, v, CT, offset):
    at, L = ctypes.c_void_p(fake.base), fake.lib
    ip, lp = P.make_params(M, K, 64, K // v, CT, 0.01)
    assert L.lutamm_load_weights(fake.ctx, 0, at, at, at, ctypes.byref(ip), ctypes.byref(lp)) == P.OK
    fake.log()
    assert L.lutamm_index_calculation(fake.ctx, 0, ctypes.c_void_p(fake.base + offset), at, ctypes.c_uint32(M), ctypes.c_uint32(P.INDEX_U8_ROWMAJOR)) == P.OK
    names = fake.log()
    assert sum("ccs_umma_kernel" in n for n in names) == tensor, names


@pytest.mark.parametrize("v,CT", [(2, 8), (2, 16), (4, 8), (4, 16), (2, 32), (8, 8)])
@pytest.mark.parametrize("M,tokens", [(16 * 65535 + 1, 4), (8 * 65535 + 1, 1), (4 * 65535 * 64 + 1, 64), (1 << 20, 1)])
def test_a_planned_run_of_the_search_fits_the_grid(fake, v, CT, M, tokens):
    """More tokens than 65535 CTAs of the planned run walk: the run grows, as the tuner tries 4 tokens at any number."""
    at, L = ctypes.c_void_p(fake.base), fake.lib
    ip, lp = P.make_params(M, 8 * v, 64, 8, CT, 0.01)
    assert L.lutamm_load_weights(fake.ctx, 0, at, at, at, ctypes.byref(ip), ctypes.byref(lp)) == P.OK
    assert L.lutamm_set_plan(fake.ctx, 0, ctypes.byref(P.Plan(ccs_tokens=tokens))) == P.OK
    fake.log()
    assert L.lutamm_index_calculation(fake.ctx, 0, at, at, ctypes.c_uint32(M), ctypes.c_uint32(P.INDEX_U8_ROWMAJOR)) == P.OK
    (line,) = fake.log()
    x, y, z = map(int, line.split()[-3:])
    assert "ccs_reg_kernel" in line and x * z == 1 and 1 <= y <= 65535


@pytest.mark.parametrize("v,CT", [(2, 16), (8, 8)])
@pytest.mark.parametrize("M", [1, 7, 4099])
@pytest.mark.parametrize("tokens", [0xFFFFFFFF, 0xFFFFFFFD, 0x80000001, 5000])
def test_a_planned_run_beyond_the_tokens(fake, v, CT, M, tokens):
    """Any number is a plan: rounded up to whole batches it stays one, and one row of CTAs takes all tokens."""
    at, L = ctypes.c_void_p(fake.base), fake.lib
    ip, lp = P.make_params(M, 8 * v, 64, 8, CT, 0.01)
    assert L.lutamm_load_weights(fake.ctx, 0, at, at, at, ctypes.byref(ip), ctypes.byref(lp)) == P.OK
    assert L.lutamm_set_plan(fake.ctx, 0, ctypes.byref(P.Plan(ccs_tokens=tokens))) == P.OK
    fake.log()
    assert L.lutamm_index_calculation(fake.ctx, 0, at, at, ctypes.c_uint32(M), ctypes.c_uint32(P.INDEX_U8_ROWMAJOR)) == P.OK
    (line,) = fake.log()
    assert "ccs_reg_kernel" in line and line.split()[-2] == "1"


@pytest.mark.parametrize("offset,kernel", [(0, "ccs_umma_kernel"), (4, "ccs_tile_kernel")])
def test_centroids_of_the_static_call_may_lie_anywhere(fake, offset, kernel):
    """The search on the tensor cores reads them 16 bytes at a time."""
    at, lib = ctypes.c_void_p(fake.base), fake.lib
    ip, lp = P.make_params(16384, 768, 64, 192, 64, 0.01)
    fake.log()
    assert lib.lutamm_amm_static_scratch(0, None, at, ctypes.c_void_p(fake.base + offset), at, at, at, ctypes.byref(ip), ctypes.byref(lp)) == P.OK
    assert kernel in fake.log()[0]


def test_the_tuner_launches_what_the_grid_holds(fake):
    """It tries runs of 4 tokens at any number of them, and a launch that fails would end it."""
    at, L = ctypes.c_void_p(fake.base), fake.lib
    M, K, N = (1 << 20) + 16, 16, 16
    ip, lp = P.make_params(M, K, N, 4, 16, 0.01)
    assert L.lutamm_load_weights(fake.ctx, 0, at, at, at, ctypes.byref(ip), ctypes.byref(lp)) == P.OK
    fake.log()
    assert L.lutamm_tune(fake.ctx, 0, ctypes.c_uint32(M), None) == P.OK
    searches = [ln for ln in fake.log() if "ccs_" in ln]
    assert len({ln for ln in searches if "ccs_reg_kernel" in ln}) > 1
    assert all(int(n) <= 65535 for ln in searches for n in ln.split()[-2:])
