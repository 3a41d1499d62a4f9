// The AMM for a few tokens: only the table rows that are used, straight from the canonical table.
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
// V > 0: the search as well, one launch for the whole operator.  A CTA searches the codebooks of its share, a thread each,
// by the reference's scan (ccs_argmin.cu) on centroids it reads itself; every column tile of a token repeats that, which
// costs less than a launch and the way of the indices through memory.
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

struct SearchArgs {
    const float *x, *centroid;   // [M][CB * V], [CB][CT][V], both 16-byte aligned
};

// The first 32 floats and then the rest of a codebook's centroids, 32 at a time: CT * V is a multiple of 4.
__device__ __forceinline__ void load_centroids(float4 (&q)[8], const float* p, uint32_t left) {
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k)
        if (4 * k < left) q[k] = __ldg(reinterpret_cast<const float4*>(p) + k);
}

// The reference's scan; q holds the first 32 floats.  32 / V centroids a batch.
template <int V>
__device__ __forceinline__ uint32_t scan(const float (&x)[V], const float* p, float4 (&q)[8], uint32_t CT) {
    float mn = 0.f;
    uint32_t best = 0;
    for (uint32_t c0 = 0; c0 < CT; c0 += 32 / V) {
        if (c0) load_centroids(q, p + c0 * V, (CT - c0) * V);
        float f[32];
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) { f[4 * k] = q[k].x; f[4 * k + 1] = q[k].y; f[4 * k + 2] = q[k].z; f[4 * k + 3] = q[k].w; }
#pragma unroll
        for (uint32_t j = 0; j < 32 / V; ++j) {
            float acc = 0.f;
#pragma unroll
            for (int d = 0; d < V; ++d) {
                const float e = __fsub_rn(x[d], f[j * V + d]);
                acc = __fadd_rn(acc, __fmul_rn(e, e));
            }
            const bool take = c0 + j == 0 || (c0 + j < CT && __fsub_rn(mn, acc) > 1e-6f);   // false for NaN: keeps the earlier index
            mn = take ? acc : mn;
            best = take ? c0 + j : best;
        }
    }
    return best;
}

template <int V>
__global__ void __launch_bounds__(kThreads, V > 0 ? 3 : 4)
lut_rows_kernel(const int8_t* __restrict__ lut, const LutArgs a, const SearchArgs sa, uint32_t per) {
    __shared__ uint32_t s_part[8][kTile / 2];
    __shared__ int32_t s_sum[kTile];
    __shared__ uint8_t s_idx[kChunk];
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5, shares = gridDim.x, rank = blockIdx.x;
    const uint32_t m = blockIdx.z, n0 = blockIdx.y * kTile;
    const uint32_t begin = rank * per, end = min(a.CB, begin + per);
    const uint32_t group = t >> 3, n = n0 + (t & 7u) * 16;
    const float bias = t < kTile && n0 + t < a.N ? __ldg(a.bias + n0 + t) : 0.f;
    float4 q[8] = {};
    if constexpr (V > 0)   // weights: nothing in the stream writes them
        if (begin + t < end) load_centroids(q, sa.centroid + (size_t)(begin + t) * a.CT * V, a.CT * V);
    pdl_wait_prior_grid();   // activations or indices, and the reader of an output that may be written again
    int32_t sum0 = 0, sum1 = 0;
    for (uint32_t c0 = begin; c0 < end; c0 += kChunk) {
        const uint32_t count = min(kChunk, end - c0);
        if constexpr (V > 0) {
            if (t < count) {
                const float* p = sa.centroid + (size_t)(c0 + t) * a.CT * V;
                float x[V];
                const float* px = sa.x + ((size_t)m * a.CB + c0 + t) * V;
                if constexpr (V == 2) {
                    const float2 u = __ldcg(reinterpret_cast<const float2*>(px));
                    x[0] = u.x; x[1] = u.y;
                } else {
#pragma unroll
                    for (int d = 0; d < V; d += 4) {
                        const float4 u = __ldcg(reinterpret_cast<const float4*>(px + d));
                        x[d] = u.x; x[d + 1] = u.y; x[d + 2] = u.z; x[d + 3] = u.w;
                    }
                }
                if (c0 != begin) load_centroids(q, p, a.CT * V);
                s_idx[t] = (uint8_t)scan<V>(x, p, q, a.CT);
            }
        } else {
            if (t < count) s_idx[t] = __ldcg(a.idx + (size_t)m * a.CB + c0 + t);
        }
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

// What a launch takes, in microseconds: 0.24 per megabyte of rows (whole tiles of columns), and rounds of CTAs; from about
// 30 MB on 0.155 per megabyte (67 MB 13 us, 134 MB 24, 268 MB 46, 537 MB 90) of a table that the half of L2 on an SM's die
// holds (of 78 MB 0.24, of 107 MB 0.44), but no less than 3 a round of CTAs.
float rows_us(uint32_t M, uint32_t CB, uint32_t CT, uint32_t N, int sm_count) {
    if (M > 65535) return 3e38f;   // a token is a block of grid.z
    const float tiles = (float)((N + kTile - 1) / kTile) * (float)M, rounds = tiles * rows_shares(M, CB, N, sm_count) / (4.f * sm_count);
    const float mb = 1e-6f * tiles * kTile * CB, few = 4.f + 0.24f * mb + (rounds > 1.f ? 1.2f * (rounds - 1.f) : 0.f), many = 6.6f + (0.155f * mb > 3.f * rounds ? 0.155f * mb : 3.f * rounds);
    return few < many || (uint64_t)CB * CT * N > 40000000 ? few : many;
}

// The same with the search, for centroid sets that a thread reads in a few batches: a lane's 16 bytes come from a line of
// their own, and a token's centroids are read once per column tile, so it goes by those bytes over all CTAs.  One launch
// over two, K = 256 to 3072, 1 to 48 tokens: where the search alone has a short form 0.8 to 0.9 up to 3 MB and 0.91 to 0.97 at 6 (v = 2,
// 16 centroids), 0.95 to 1.05 at 7, 1.08 to 1.17 at 9; with 128 floats a codebook (v = 8, 16) 0.97 at 10.6, 1.00 to 1.18 at 14; where it has none
// (v = 4, 13 centroids) 0.83 at 15, 0.96 to 1.05 at 23, (v = 4, 32) 0.82 to 1.01 at 14, 1.14 at 17.
bool rows_search_ok(uint32_t M, uint32_t CB, uint32_t CT, uint32_t v, uint32_t N, const float* x) {
    if ((v != 2 && v != 4 && v != 8) || CT * v % 4 || CT * v > 128 || (reinterpret_cast<uintptr_t>(x) & 15u) || (uint64_t)CB * v % 4) return false;
    const uint64_t most = !ccs_has_short_form(v, CT) ? 16000000 : CT * v > 64 ? 13000000 : 6500000;
    return (uint64_t)M * ((N + kTile - 1) / kTile) * CB * CT * v * 4 <= most;
}

template <int V>
static cudaError_t run_rows(const LutArgs& a, const int8_t* lut, const SearchArgs& sa, int sm_count, cudaStream_t s) {
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
    return cudaLaunchKernelEx(&cfg, lut_rows_kernel<V>, lut, a, sa, per);
}

cudaError_t launch_rows(const LutArgs& a, const int8_t* lut, int sm_count, cudaStream_t s) {
    if (a.M == 0 || a.N == 0) return cudaSuccess;
    return run_rows<0>(a, lut, SearchArgs{}, sm_count, s);
}

cudaError_t launch_rows_search(const LutArgs& a, const int8_t* lut, const float* x, const float* centroid, uint32_t v, int sm_count, cudaStream_t s) {
    if (a.M == 0 || a.N == 0) return cudaSuccess;
    const SearchArgs sa{x, centroid};
    return v == 2 ? run_rows<2>(a, lut, sa, sm_count, s) : v == 4 ? run_rows<4>(a, lut, sa, sm_count, s) : run_rows<8>(a, lut, sa, sm_count, s);
}

}  // namespace lutamm
