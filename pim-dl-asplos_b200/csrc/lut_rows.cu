// Steps 2+3 of the AMM for a few tokens: only the table rows that are used, straight from the canonical table.
//
// The contraction kernels read the whole table whatever the number of tokens; M tokens use M of a codebook's CT rows at
// most.  Up to that many bytes, M * CB * N against CB * CT * N, it is cheaper to fetch rows: 9 tokens through 3328
// codebooks of 16 -> 1152 are 35 MB instead of 61.
//
// A CTA takes one token, 128 columns and a share of the codebooks: 8 lanes per row, 16 bytes each, so a warp reads four
// rows and every thread has 8 loads in flight.  Bytes are widened to 16 bits, two per register, offset by 128 so that
// they cannot be negative: 256 rows of at most 255 fit, which is what a CTA reduces before it adds to int32.  The CTAs
// of a cluster hold the shares of one token and tile and are summed through distributed shared memory.
//
// What bounds it: launch and a chain of three latencies (index, row, cluster) up to about 10 MB of rows, L2 above (31 MB
// in 11.4 us).  Against the contraction: 32 tokens, 384 codebooks of 16 -> 768 8.3 -> 5.4 us; one token, 1616 codebooks of
// 32 -> 1984 27.5 -> 4.4 us; 16 tokens, 256 codebooks of 128 -> 4016 33 -> 4.7 us.
#include "kernels.h"
#include "ptx.cuh"
#include "epilogue.cuh"

namespace lutamm {

namespace {

constexpr uint32_t kThreads = 256, kTile = 128, kChunk = 256;   // columns of a CTA, codebooks between int32 sums
constexpr uint32_t kMaxCluster = 8;

__device__ __forceinline__ int32_t load_cluster(uint32_t addr) {
    int32_t v;
    asm volatile("ld.shared::cluster.b32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}

__global__ void __launch_bounds__(kThreads, 4)
lut_rows_kernel(const int8_t* __restrict__ lut, const LutArgs a, uint32_t per) {
    __shared__ uint32_t s_part[8][kTile / 2];
    __shared__ int32_t s_sum[kTile];
    __shared__ uint8_t s_idx[kChunk];
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5, shares = gridDim.x, rank = blockIdx.x;
    const uint32_t m = blockIdx.z, n0 = blockIdx.y * kTile;
    const uint32_t begin = rank * per, end = min(a.CB, begin + per);
    const uint32_t group = t >> 3, n = n0 + (t & 7u) * 16;
    const float bias = t < kTile && n0 + t < a.N ? __ldg(a.bias + n0 + t) : 0.f;
    pdl_wait_prior_grid();   // indices, and the reader of an output that may be written again
    int32_t sum0 = 0, sum1 = 0;
    for (uint32_t c0 = begin; c0 < end; c0 += kChunk) {
        const uint32_t count = min(kChunk, end - c0);
        if (t < count) s_idx[t] = __ldcg(a.idx + (size_t)m * a.CB + c0 + t);
        __syncthreads();
        uint4 w[8];
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) {
            const uint32_t c = group + 32 * j;
            w[j] = make_uint4(0, 0, 0, 0);
            if (c < count && n < a.N) {
                const uint32_t i = s_idx[c];   // one that is out of range adds nothing
                if (i < a.CT) w[j] = __ldg(reinterpret_cast<const uint4*>(lut + ((size_t)(c0 + c) * a.CT + i) * a.N + n));
            }
        }
        uint32_t acc[8] = {};   // [word][columns 0 and 2, columns 1 and 3]
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) {
            const uint32_t q[4] = {w[j].x, w[j].y, w[j].z, w[j].w};
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) {
                acc[2 * k] += (q[k] ^ 0x80808080u) & 0x00FF00FFu;
                acc[2 * k + 1] += ((q[k] >> 8) ^ 0x00808080u) & 0x00FF00FFu;
            }
        }
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
            acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], 8);
            acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], 16);
        }
        if (lane < 8) {
#pragma unroll
            for (uint32_t k = 0; k < 8; k += 4)
                *reinterpret_cast<uint4*>(&s_part[warp][lane * 8 + k]) = make_uint4(acc[k], acc[k + 1], acc[k + 2], acc[k + 3]);
        }
        __syncthreads();
        if (t < kTile / 2) {
            uint32_t s = 0;
#pragma unroll
            for (uint32_t k = 0; k < 8; ++k) s += s_part[k][t];
            sum0 += (int32_t)(s & 0xFFFFu) - 128 * (int32_t)kChunk;   // every thread added 8 rows, some of them zero
            sum1 += (int32_t)(s >> 16) - 128 * (int32_t)kChunk;
        }
    }
    if (t < kTile / 2) {
        const uint32_t col = (t >> 3) * 16 + ((t >> 1) & 3u) * 4 + (t & 1u);
        s_sum[col] = sum0;
        s_sum[col + 2] = sum1;
    }
    if (shares > 1) cluster_sync(); else __syncthreads();
    if (rank == 0 && t < kTile && n0 + t < a.N) {
        int32_t acc = s_sum[t];
        for (uint32_t r = 1; r < shares; ++r) acc += load_cluster(map_to_rank(smem_u32(s_sum + t), r));
        const float y = dequant_one(acc, a.scale, lut_bias_times_cb(a.lut_bias, a.CB), bias);
        a.out[(size_t)m * a.N + n0 + t] = activate_one(y, a.act);
    }
    if (shares > 1) cluster_sync();   // the sums are read
}

}  // namespace

// Shares of the codebook axis: until the SMs have a CTA and a half each, at most one cluster, of 32 codebooks at least.
// (A launch is done in 4.5 us without a cluster and in 5.3 with one; 8 tokens, 1536 codebooks -> 768: 11.9 us whole, 8.8 in
// halves, 7.9 in quarters, 7.0 in eighths.)
static uint32_t rows_shares(uint32_t M, uint32_t CB, uint32_t N, int sm_count) {
    const uint64_t tiles = (uint64_t)M * ((N + kTile - 1) / kTile);
    uint32_t shares = 1;
    while (shares < kMaxCluster && 2 * tiles * shares < 3ull * sm_count && shares * 64 <= CB) shares *= 2;
    return shares;
}

// What a launch takes, in microseconds: 0.24 per megabyte of rows (whole tiles of columns), and rounds of CTAs.
float rows_us(uint32_t M, uint32_t CB, uint32_t N, int sm_count) {
    const float tiles = (float)((N + kTile - 1) / kTile) * (float)M, rounds = tiles * rows_shares(M, CB, N, sm_count) / (4.f * sm_count);
    return 4.f + 0.24e-6f * tiles * kTile * CB + (rounds > 1.f ? 1.2f * (rounds - 1.f) : 0.f);
}

cudaError_t launch_rows(const LutArgs& a, const int8_t* lut, int sm_count, cudaStream_t s) {
    if (a.M == 0 || a.N == 0) return cudaSuccess;
    const uint32_t shares = rows_shares(a.M, a.CB, a.N, sm_count), per = (a.CB + shares - 1) / shares;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(shares, (a.N + kTile - 1) / kTile, a.M);
    cfg.blockDim = dim3(kThreads);
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = shares;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, lut_rows_kernel, lut, a, per);
}

}  // namespace lutamm
