// The AMM for a few tokens: only the table rows that are used, straight from the canonical table.
//
// The contraction kernels read the whole table whatever the number of tokens; M tokens use M of a codebook's CT rows at
// most.  Up to that many bytes, M * CB * N against CB * CT * N, it is cheaper to fetch rows: 9 tokens through 3328
// codebooks of 16 -> 1152 are 35 MB instead of 61.
//
// A CTA takes one token, 128 columns and a share of the codebooks: 8 lanes per row, 16 bytes each, so a warp reads four
// rows and every thread has 8 loads in flight, a chunk of 256 codebooks; the indices of the next chunk are on their way
// meanwhile.  Bytes are widened to 16 bits, two per register, offset by 128 so that they cannot be negative: 256 rows of at
// most 255 fit into what four threads of a warp add up, so warps meet and add to int32 once in 8 chunks (once in every
// chunk 1536 codebooks -> 768 took 10.9 us for one token, and 9.5 now).  The CTAs of a cluster hold the shares of one token and
// tile and are summed through distributed shared memory.
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

constexpr uint32_t kThreads = 256, kTile = 128, kChunk = 256;   // columns of a CTA, codebooks whose rows are in flight together
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

// LONG: shares of more than one chunk.  (One kernel for both cost calls of one chunk 0.4 us of 3.8.)
template <int V, bool LONG>
__global__ void __launch_bounds__(kThreads, V > 0 ? (LONG ? 2 : 3) : 4)
lut_rows_kernel(const int8_t* __restrict__ lut, const LutArgs a, const SearchArgs sa, uint32_t per) {
    __shared__ uint32_t s_part[8][kTile / 2];
    __shared__ int32_t s_sum[kTile];
    __shared__ uint8_t s_idx[LONG ? 2 : 1][kChunk];
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
    uint32_t acc[8] = {}, buf = 0, pending = 0;   // [word][columns 0 and 2, columns 1 and 3]; chunks in it
    uint8_t ahead = 0;   // this thread's index of the next chunk
    if (LONG && V == 0 && begin + t < end) ahead = __ldcg(a.idx + (size_t)m * a.CB + begin + t);
    uint32_t c0 = begin;
    do {
        const uint32_t count = c0 < end ? min(kChunk, end - c0) : 0u;
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
                if (LONG && c0 != begin) load_centroids(q, p, a.CT * V);
                s_idx[buf][t] = (uint8_t)scan<V>(x, p, q, a.CT);
            }
        } else {
            if constexpr (LONG) {
                s_idx[buf][t] = ahead;
                if (c0 + kChunk + t < end) ahead = __ldcg(a.idx + (size_t)m * a.CB + c0 + kChunk + t);
            } else {
                if (t < count) s_idx[0][t] = __ldcg(a.idx + (size_t)m * a.CB + c0 + t);
            }
        }
        __syncthreads();
        uint4 w[8];
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) {
            const uint32_t c = group + 32 * j;
            w[j] = make_uint4(0, 0, 0, 0);
            if (c < count && n < a.N) {
                const uint32_t i = s_idx[buf][c];   // one that is out of range adds nothing
                if (i < a.CT) w[j] = __ldg(reinterpret_cast<const uint4*>(lut + ((size_t)(c0 + c) * a.CT + i) * a.N + n));
            }
        }
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) {
            const uint32_t q[4] = {w[j].x, w[j].y, w[j].z, w[j].w};
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) {
                acc[2 * k] += (q[k] ^ 0x80808080u) & 0x00FF00FFu;
                acc[2 * k + 1] += ((q[k] >> 8) ^ 0x00808080u) & 0x00FF00FFu;
            }
        }
        if constexpr (LONG) {
            buf ^= 1;
            c0 += kChunk;
            if (++pending < 8 && c0 < end) continue;
        }
        // 64 rows of a thread at most, over the four threads of a warp that hold the same columns: 256 * 255 < 2^16
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
            const int32_t none = -128 * (int32_t)((LONG ? pending : 1) * kChunk);   // a row, or the zero in its place, was added with 128 more
            sum0 += none;
            sum1 += none;
            if (!LONG || pending == 1) {   // 8 rows a thread: all 256 fit into the two halves
                uint32_t s = 0;
#pragma unroll
                for (uint32_t k = 0; k < 8; ++k) s += s_part[k][t];
                sum0 += (int32_t)(s & 0xFFFFu);
                sum1 += (int32_t)(s >> 16);
            } else {
#pragma unroll
                for (uint32_t k = 0; k < 8; ++k) {
                    const uint32_t s = s_part[k][t];
                    sum0 += (int32_t)(s & 0xFFFFu);
                    sum1 += (int32_t)(s >> 16);
                }
            }
        }
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) acc[k] = 0;
        pending = 0;
    } while (LONG && c0 < end);
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

// What a call takes, in microseconds, with its codebook axis in `shares`: a cluster is a microsecond, so is every chunk of
// codebooks after the first (two where they are searched, too), a CTA costs 4 ns and its rows 11 ns per 1000, and a table
// that the half of L2 on an SM's die does not hold costs more per row.  With the search every CTA also reads and scans the
// centroids of its share.  Fitted to 870 calls of 1 to 200 tokens, 256 to 8192 features, 5 to 128 centroids, each with 1, 2, 4
// and 8 shares, to 20 % (11 % with the search).  By the least of these, and of the contraction in lutamm_capi.cu, those calls
// take 0.7 % more than the fastest form of each; 5.5 % with as many shares as made a CTA and a half for every SM.
static float rows_call_us(bool search, uint32_t M, uint32_t CB, uint32_t CT, uint32_t v, uint32_t N, uint32_t shares, int sm_count) {
    const uint32_t per = (CB + shares - 1) / shares;
    const float tiles = (float)((N + kTile - 1) / kTile) * (float)M, ctas = tiles * shares * (148.f / sm_count), more = (float)((per + kChunk - 1) / kChunk - 1);
    const float far = (uint64_t)CB * CT * N > 40000000 ? 1e-6f * tiles * kTile * CB : 0.f, cluster = shares > 1 ? 1.f : 0.f;
    if (search)
        return 2.1f + cluster * (1.f + 0.00043f * ctas * shares) + 0.0039f * ctas + 12.6e-6f * ctas * per + 0.022f * far +
               more * (1.9f + 0.0066f * CT * v) + 1.5e-4f * (per < kChunk ? per : kChunk) * CT * v + 5e-7f * tiles * CB * CT * v;
    return 4.5f + cluster * (1.1f + 0.00032f * ctas * shares) + 0.0003f * per + 0.0038f * ctas + 11.4e-6f * ctas * per + 0.032f * far + 1.1f * more;
}

// The split of the codebook axis, at least 32 codebooks a CTA.  8 tokens, 384 codebooks of 16 -> 768 with the search: eighths
// 5.25 us, halves 4.4, whole 5.8; 32 tokens without: whole 5.9, halves 6.5.
static uint32_t rows_shares(bool search, uint32_t M, uint32_t CB, uint32_t CT, uint32_t v, uint32_t N, int sm_count) {
    uint32_t best = 1;
    float least = rows_call_us(search, M, CB, CT, v, N, 1, sm_count);
    for (uint32_t s = 2; s <= kMaxCluster && s * 32 <= CB; s *= 2) {
        const float us = rows_call_us(search, M, CB, CT, v, N, s, sm_count);
        if (us < least) { least = us; best = s; }
    }
    return best;
}

// Without the search, which the other forms need as well.
float rows_us(uint32_t M, uint32_t CB, uint32_t CT, uint32_t N, int sm_count) {
    if (M > 65535) return 3e38f;   // a token is a block of grid.z
    return rows_call_us(false, M, CB, CT, 0, N, rows_shares(false, M, CB, CT, 0, N, sm_count), sm_count);
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
    const uint32_t shares = rows_shares(V > 0, a.M, a.CB, a.CT, V, a.N, sm_count), per = (a.CB + shares - 1) / shares;
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
    return cudaLaunchKernelEx(&cfg, per > kChunk ? lut_rows_kernel<V, true> : lut_rows_kernel<V, false>, lut, a, sa, per);
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
