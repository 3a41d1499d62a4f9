"""lutamm_build_lut's two launches with a runtime that refuses one of them: the maximum that pass 1 leaves must not scale
the next table.  The object file of the library, linked with a stand-in for the CUDA runtime: no GPU."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pim-dl-asplos_b200", "csrc")
OBJECT = os.path.join(CSRC, "build", "lut_build.o")
INCLUDE = "/usr/local/cuda/include"

FAKE = r"""
#include "kernels.h"
#include <cstdio>
#include <cstring>

static int launches, refuse, cleared;
static cudaError_t pending = cudaSuccess;
static uint32_t words[2] = {0, 0};

static cudaError_t launch() {
    if (launches++ == refuse) return pending = cudaErrorLaunchOutOfResources;
    if (launches == 1) words[0] = 0x42000000u;   // what pass 1 would find
    else words[0] = words[1] = 0;                // and pass 2 re-arm
    return cudaSuccess;
}

extern "C" {
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return launch(); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**) { return launch(); }
cudaError_t cudaGetLastError() { const cudaError_t e = pending; pending = cudaSuccess; return e; }
cudaError_t cudaMemsetAsync(void* p, int value, size_t bytes, cudaStream_t) { std::memset(p, value, bytes); ++cleared; return cudaSuccess; }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
}

int main(int argc, char** argv) {
    refuse = argv[1][0] - '0';
    alignas(16) static float weight[64];
    static float scalars[2], centroid[64];
    alignas(4) static int8_t lut[256];
    lutamm::LutBuildArgs a{centroid, weight, lut, words, scalars, 2, 8, argc > 2 ? 3u : 2u, 16};
    const char* why = nullptr;
    const cudaError_t e = lutamm::launch_lut_build(a, nullptr, &why);
    std::printf("%d %d %u %u\n", (int)e, launches, words[0], words[1]);
    return 0;
}
"""


@pytest.mark.skipif(not (os.path.exists(OBJECT) and shutil.which("g++") and os.path.exists(os.path.join(INCLUDE, "cuda_runtime.h"))),
                    reason="the library's objects or the toolkit's headers are not here")
def test_a_refused_launch_leaves_no_maximum_behind(tmp_path):
    (tmp_path / "fake.cpp").write_text(FAKE)
    exe = str(tmp_path / "fake")
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-I", INCLUDE, "-o", exe, str(tmp_path / "fake.cpp"), OBJECT], check=True, timeout=120)
    for more in ([], ["run-time length"]):
        code, launches, maximum, blocks = map(int, subprocess.run([exe, "9"] + more, capture_output=True, text=True, check=True).stdout.split())
        assert (code, launches, maximum, blocks) == (0, 2, 0, 0)
        code, launches, maximum, blocks = map(int, subprocess.run([exe, "1"] + more, capture_output=True, text=True, check=True).stdout.split())
        assert code != 0 and launches == 2 and (maximum, blocks) == (0, 0)
        code, launches, maximum, blocks = map(int, subprocess.run([exe, "0"] + more, capture_output=True, text=True, check=True).stdout.split())
        assert code != 0 and launches == 1 and (maximum, blocks) == (0, 0)   # pass 2 has nothing to read
