// Load-time construction of a layer's int8 lookup table from its centroids and its dense
// weight: what model-calibration/pim_weight_converter.py:21-36,83-91 of the reference does with
// torch.bmm + lut_quant, as two passes that never materialise the fp32 table.
//
//   lut_f[cb][ct][n] = sum_d centroid[cb][ct][d] * weight[cb*v + d][n]     (fp32, d ascending, unfused)
//   scale            = max|lut_f| / 127                                    (zero point 0)
//   lut[cb][ct][n]   = int8( rint( clamp( lut_f / scale, -128, 127 ) ) )   (round half to even)
//
// Pass 1 reduces max|lut_f|; pass 2 recomputes the products and writes the bytes.  Compulsory
// traffic: the weight twice (8*K*N bytes) plus the table once (CB*CT*N bytes).
//
// What bounds it: while an SM has blocks, dispatch (pass 2 at v = 2: twelve lane instructions a table byte, issue in 72 % of
// the cycles); of a launch over 18.9 MB of table that is 58 %, the rest is the launch, each block's chain of centroids, barrier
// and weights, and blocks that end apart.  The quotient is rounded by one packed
// multiply-add to a number whose low mantissa byte is the result, and only a value within 5e-5 of a half-way point
// (the reciprocal's error is below 2e-5) is divided; the two scalars go straight to mapped host memory and the maximum is
// re-armed by the last block, so that a call is two launches and a wait.  BERT-base FFN1 (18.9 MB of table): pass 2
// 18.6 -> 13.8 us from a cold L2, the call 59 -> 30 us.
#include "kernels.h"
#include "ptx.cuh"

namespace lutamm {
namespace {

constexpr int kThreads = 256;
constexpr uint32_t kTogether = 8;
constexpr int kMaxV = 1024;  // run-time path; bounded by the shared-memory check below

// The products and sums, each rounded on its own.  Scalar on purpose: a packed multiplication followed by a packed
// addition came out of the compiler fused, explicit rounding or not.
__device__ __forceinline__ float2 times(float c, float2 w) { return make_float2(__fmul_rn(c, w.x), __fmul_rn(c, w.y)); }
__device__ __forceinline__ float2 plus(float2 a, float2 b) { return make_float2(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y)); }

// One block: one codebook x one chunk of kThreads*4 output columns.  A thread owns four
// adjacent columns (one 16-byte weight load per sub-vector dimension, one 4-byte table
// store per centroid, so a warp writes 128 contiguous bytes per centroid row).
// V > 0: compile-time sub-vector length, the thread's weight slice lives in registers.
// V == 0: run-time length, the slice is re-read (L1 resident) for every kTogether centroids; one at a time the load was
// most of what a sum took (4160 x 8368, v = 20: 330 -> 191 us a call).  In registers a call is 1.2 to 1.7 times as fast, at 32
// too, where they leave room for one block an SM: 5120 x 16384, 16 centroids, v = 10 398 -> 241 us, v = 20 359 -> 246, v = 32
// 352 -> 297; 640 x 2560 34 -> 28, 39 -> 29, 49 -> 31.
template <int V, bool kWrite>
__global__ void __launch_bounds__(kThreads)
lut_build_kernel(const float* __restrict__ centroid, const float* __restrict__ weight, int8_t* __restrict__ lut,
                 uint32_t* __restrict__ words, float* __restrict__ scalars, uint32_t CT, uint32_t v_rt, uint32_t N) {
    extern __shared__ float s_cent[];  // [CT][v]
    if (!kWrite) pdl_launch_dependents();   // pass 2 stages its operands meanwhile
    const uint32_t v = V > 0 ? (uint32_t)V : v_rt;
    const uint32_t cb = blockIdx.y;
    for (uint32_t i = threadIdx.x; i < CT * v; i += kThreads) s_cent[i] = centroid[(size_t)cb * CT * v + i];

    const uint32_t n0 = (blockIdx.x * kThreads + threadIdx.x) * 4;
    const float* wrow = weight + (size_t)cb * v * N + n0;
    float2 w[V > 0 ? V : 1][2];
    if (V > 0 && n0 < N) {
#pragma unroll
        for (int d = 0; d < V; ++d) {
            const float4 t = __ldg(reinterpret_cast<const float4*>(wrow + (size_t)d * N));
            w[d][0] = make_float2(t.x, t.y); w[d][1] = make_float2(t.z, t.w);
        }
    }
    __syncthreads();
    float scale = 1.f, inv_scale = 1.f;
    if (kWrite) {
        pdl_wait_prior_grid();
        scale = __fdiv_rn(__uint_as_float(__ldcg(words)), 127.f);
        inv_scale = __fdiv_rn(1.f, scale);
    }
    float amax = 0.f;
    if (n0 < N) {
        auto finish = [&](uint32_t ct, const float2 (&a)[2]) {
            if (!kWrite) {
                amax = fmaxf(amax, fmaxf(fmaxf(fabsf(a[0].x), fabsf(a[0].y)), fmaxf(fabsf(a[1].x), fabsf(a[1].y))));
            } else {
                // t = x / scale + 1.5 * 2^23: its low mantissa bits are the rounded quotient, its distance from x / scale
                // tells how close to half-way that was (NaN and infinity do not compare)
                constexpr float kMagic = 12582912.f;
                const float2 inv2 = make_float2(inv_scale, inv_scale);
                float2 t[2], off[2];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    t[k] = __ffma2_rn(a[k], inv2, make_float2(kMagic, kMagic));
                    const float2 n = __fadd2_rn(t[k], make_float2(-kMagic, -kMagic));
                    off[k] = __ffma2_rn(a[k], inv2, make_float2(-n.x, -n.y));
                }
                const float far = fmaxf(fmaxf(fabsf(off[0].x), fabsf(off[0].y)), fmaxf(fabsf(off[1].x), fabsf(off[1].y)));
                const bool number = fabsf(off[0].x + off[0].y + off[1].x + off[1].y) <= 2.f;
                uint32_t bytes = __byte_perm(__byte_perm(__float_as_uint(t[0].x), __float_as_uint(t[0].y), 0x0040),
                                             __byte_perm(__float_as_uint(t[1].x), __float_as_uint(t[1].y), 0x0040), 0x5410);
                if (!(far < 0.49995f && number)) {
                    auto q = [scale](float x) -> uint32_t { return (uint32_t)(int)rintf(fminf(fmaxf(__fdiv_rn(x, scale), -128.f), 127.f)) & 0xFFu; };
                    bytes = scale > 0.f ? q(a[0].x) | q(a[0].y) << 8 | q(a[1].x) << 16 | q(a[1].y) << 24
                                        : 0u;  // an all-zero table has no scale; the reference would emit NaN bytes
                }
                *reinterpret_cast<uint32_t*>(lut + ((size_t)cb * CT + ct) * N + n0) = bytes;
            }
        };
        // products and sums rounded one by one, ascending; 0 + c w is c w (but for the sign of a zero)
        if constexpr (V > 0) {
            for (uint32_t ct = 0; ct < CT; ++ct) {
                float2 a[2];
#pragma unroll
                for (int d = 0; d < V; ++d) {
                    const float c = s_cent[ct * V + d];
#pragma unroll
                    for (int k = 0; k < 2; ++k) a[k] = d == 0 ? times(c, w[d][k]) : plus(a[k], times(c, w[d][k]));
                }
                finish(ct, a);
            }
        } else {
            for (uint32_t ct0 = 0; ct0 < CT; ct0 += kTogether) {
                float2 a[kTogether][2];
#pragma unroll
                for (uint32_t j = 0; j < kTogether; ++j) a[j][0] = a[j][1] = make_float2(0.f, 0.f);
                const float* cent[kTogether];
#pragma unroll
                for (uint32_t j = 0; j < kTogether; ++j) cent[j] = s_cent + min(ct0 + j, CT - 1) * v;
                for (uint32_t d = 0; d < v; ++d) {
                    const float4 t = __ldg(reinterpret_cast<const float4*>(wrow + (size_t)d * N));
#pragma unroll
                    for (uint32_t j = 0; j < kTogether; ++j) {
                        const float c = cent[j][d];
                        a[j][0] = plus(a[j][0], times(c, make_float2(t.x, t.y)));
                        a[j][1] = plus(a[j][1], times(c, make_float2(t.z, t.w)));
                    }
                }
#pragma unroll
                for (uint32_t j = 0; j < kTogether; ++j)
                    if (ct0 + j < CT) finish(ct0 + j, a[j]);
            }
        }
    }
    if (!kWrite) {
        // non-negative floats order like their bit patterns
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        __shared__ float s_w[kThreads / 32];
        if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = amax;
        __syncthreads();
        if (threadIdx.x == 0) {
            float m = s_w[0];
            for (int i = 1; i < kThreads / 32; ++i) m = fmaxf(m, s_w[i]);
            if (m == m) atomicMax(words, __float_as_uint(m));
        }
    } else {
        __syncthreads();
        // every block has read the maximum before it counts itself here: the last one clears it for the next call
        if (threadIdx.x == 0 && atomicAdd(words + 1, 1u) == gridDim.x * gridDim.y - 1) {
            words[0] = 0u;
            words[1] = 0u;
            scalars[0] = scale;
            scalars[1] = -scale * 0.f;  // -scale * zero_point, zero_point = 0 (pim_weight_converter.py:35)
            __threadfence_system();
        }
    }
}

template <int V>
cudaError_t launch_both(const LutBuildArgs& a, dim3 grid, size_t smem, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaError_t e = cudaLaunchKernelEx(&cfg, lut_build_kernel<V, false>, a.centroid, a.weight, static_cast<int8_t*>(nullptr), a.words, static_cast<float*>(nullptr), a.CT, a.v, a.N);
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, lut_build_kernel<V, true>, a.centroid, a.weight, a.lut, a.words, a.scalars, a.CT, a.v, a.N);
    // only pass 2 clears the maximum that pass 1 leaves, and the next table would be scaled with it
    if (e != cudaSuccess) cudaMemsetAsync(a.words, 0, 2 * sizeof(uint32_t), s);
    return e;
}

}  // namespace

// The reference keeps the LUT it sends to the DPUs re-tiled along the output features
// (reorder_pim_lut, inference-engine/test/test_amm.cpp:71-121):
//   dpu[(f / T) * rows * T + row * T + f % T] = canonical[row * N + f],   row = cb * CT + ct,
// T = feature_stile_size (STATIC load type) or feature_load_tile_size (FINE / COARSE).  This
// turns such a table back into the canonical [CB][CT][N] layout the kernels read.
namespace {
__global__ void lut_untile_kernel(const int8_t* __restrict__ dpu, int8_t* __restrict__ canonical, uint32_t rows,
                                  uint32_t N, uint32_t T) {
    const uint32_t row = blockIdx.y;
    for (uint32_t f = blockIdx.x * blockDim.x + threadIdx.x; f < N; f += gridDim.x * blockDim.x)
        canonical[(size_t)row * N + f] = dpu[(size_t)(f / T) * rows * T + (size_t)row * T + f % T];
}
}  // namespace

cudaError_t launch_lut_untile(const int8_t* dpu, int8_t* canonical, uint32_t rows, uint32_t N, uint32_t T,
                              cudaStream_t s, const char** why) {
    *why = nullptr;
    if (T == 0 || N % T != 0) { *why = "output_feature_len must be a multiple of the LUT tile width"; return cudaErrorInvalidValue; }
    if (rows == 0 || rows > 65535u * 32u) { *why = "LUT has too many rows"; return cudaErrorInvalidValue; }
    // rows can exceed the 65535 limit of grid.y: fold the excess into a loop over row blocks
    const uint32_t per = 65535u;
    for (uint32_t r0 = 0; r0 < rows; r0 += per) {
        const uint32_t nr = rows - r0 < per ? rows - r0 : per;
        const dim3 grid((N + 255) / 256 > 64 ? 64 : (N + 255) / 256, nr);
        // the tile term of the source index uses the full row count, the row term the absolute row
        lut_untile_kernel<<<grid, 256, 0, s>>>(dpu + (size_t)r0 * T, canonical + (size_t)r0 * N, rows, N, T);
    }
    return cudaGetLastError();
}

cudaError_t launch_lut_build(const LutBuildArgs& a, cudaStream_t s, const char** why) {
    *why = nullptr;
    if (a.v == 0 || a.v > kMaxV) { *why = "sub-vector length must be 1..1024"; return cudaErrorInvalidValue; }
    if (a.CB == 0 || a.CB > 65535 || a.CT == 0) { *why = "num_codebook must be 1..65535 and num_centroid non-zero"; return cudaErrorInvalidValue; }
    if (a.N % 4 != 0) { *why = "output features must be a multiple of 4"; return cudaErrorInvalidValue; }
    if ((reinterpret_cast<uintptr_t>(a.weight) & 15) || (reinterpret_cast<uintptr_t>(a.lut) & 3)) {
        *why = "weight must be 16-byte aligned, table 4-byte aligned"; return cudaErrorInvalidValue;
    }
    const size_t smem = (size_t)a.CT * a.v * sizeof(float);
    if (smem > 48 * 1024) { *why = "centroids of one codebook exceed 48 KB"; return cudaErrorInvalidValue; }
    const dim3 grid((a.N / 4 + kThreads - 1) / kThreads, a.CB);
    cudaError_t e;
    switch (a.v) {
        case 1: e = launch_both<1>(a, grid, smem, s); break;
        case 2: e = launch_both<2>(a, grid, smem, s); break;
        case 4: e = launch_both<4>(a, grid, smem, s); break;
        case 8: e = launch_both<8>(a, grid, smem, s); break;
        case 10: e = launch_both<10>(a, grid, smem, s); break;
        case 16: e = launch_both<16>(a, grid, smem, s); break;
        case 20: e = launch_both<20>(a, grid, smem, s); break;
        case 32: e = launch_both<32>(a, grid, smem, s); break;
        default: e = launch_both<0>(a, grid, smem, s); break;
    }
    return e == cudaSuccess ? cudaGetLastError() : e;
}

}  // namespace lutamm
