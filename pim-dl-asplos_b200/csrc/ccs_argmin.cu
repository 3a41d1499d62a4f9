// Step 1 of the AMM: closest-centroid search (CCS).
//
// Replaces index_calculation() of the reference (inference-engine/src/host/index_calc_host.cpp:8-53).
// The result has to match that function bit for bit.  There
//   * every fp32 operation rounds on its own (the reference is built for baseline x86-64, no FMA);
//   * the squared distance accumulates in dimension order starting from 0;
//   * the "argmin" is a sequential scan with hysteresis - centroid c replaces the running minimum only
//     if fl(min - dist[c]) > 1e-6 - so near-ties are decided by the order of the scan.
//
// exact_scan() (ccs_scan.cuh) is that statement, one (token, codebook) in one thread, ~3v + 4 instructions per centroid.
// It runs only where it can matter.  Every (token, codebook) first goes through a FILTER that evaluates
//     s_c = |c|^2 / 2 - x.c      (so that |x - c|^2 = |x|^2 + 2 s_c),   v fused multiply-adds per centroid,
// and looks for centroids within a margin T of the smallest s_c.  If there is exactly one, the scan ends on it
// whatever the order: with D_c the true squared distance, A = |x|^2, B = max |c|^2 and u = 2^-24,
//     |s_c computed - s_c|       <= 1.01 (2v+1) u (A + B)
//     |dist[c] computed - D_c|   <= 1.01 (v+3) u D_c,   and D of the winner <= 2 (A + B),
// so a gap of more than T = 0.51e-6 + (8v + 16) u (A + B) in s makes fl(dist[c] - dist[winner]) > 1e-6 for
// every other c: the scan takes the winner when it meets it and nothing after it.  Otherwise - two candidates,
// or anything not finite - the thread runs exact_scan.  For N(0,1) data a few scans in 1e5 do at v = 2.
//
// What bounds it: dispatch, in ccs_reg_kernel.  Per centroid v/2 packed multiply-adds, half a packed addition (two
// dispatch cycles each), half a three-input minimum and a funnel shift that collects the comparison's sign bit, against
// 3v/2 packed and 4 other instructions of the scan; per (token, codebook) about 25 instructions around that.
// 65536 x 2048 codebooks, v = 2, 16 centroids: 442 us (the scan alone 593), the ALU pipe 53 % and the FMA pipe 45 % busy
// (they hardly overlap).  ccs_tile_kernel issues in 40 to 60 % of the cycles: a CTA stages everything, waits, and computes.
//
// Calls of many scores take the filter to the tensor cores: ccs_umma.cu.
//
// Two mappings:
//   ccs_reg_kernel  thread <-> codebook, the codebook's centroids in registers, the thread walks a run of
//                   tokens; activations load as coalesced float2 / float4.  Small centroid sets.
//   ccs_tile_kernel thread <-> token (one or two), activations and centroids of a few codebooks staged in
//                   shared memory, a centroid is read as a warp-wide broadcast.  Any v up to 32, any CT.
//   ccs_any_kernel  any v, exact_scan alone.
//
// HBM traffic: 4*M*K (activations) + 4*CB*CT*v (centroids) + M*CB (uint8 indices).
#include "kernels.h"
#include "ccs_scan.cuh"
#include "../../include/lutamm.h"
#include <algorithm>

namespace lutamm {

namespace {

// V floats of shared memory
template <int V>
__device__ __forceinline__ void load_x(const float* p, float (&f)[V]) {
    if constexpr (V % 4 == 0) {
#pragma unroll
        for (int i = 0; i < V / 4; ++i) {
            const float4 t = *reinterpret_cast<const float4*>(p + 4 * i);
            f[4 * i + 0] = t.x; f[4 * i + 1] = t.y; f[4 * i + 2] = t.z; f[4 * i + 3] = t.w;
        }
    } else if constexpr (V % 2 == 0) {
#pragma unroll
        for (int i = 0; i < V / 2; ++i) {
            const float2 t = *reinterpret_cast<const float2*>(p + 2 * i);
            f[2 * i + 0] = t.x; f[2 * i + 1] = t.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < V; ++i) f[i] = p[i];
    }
}

// V floats of global memory
template <int V>
__device__ __forceinline__ void load_global(const float* __restrict__ p, float (&f)[V]) {
    static_assert(V == 2 || V % 4 == 0, "vector loads");
    if constexpr (V == 2) {
        const float2 t = __ldg(reinterpret_cast<const float2*>(p));
        f[0] = t.x; f[1] = t.y;
    } else {
#pragma unroll
        for (int i = 0; i < V; i += 4) {
            const float4 t = __ldg(reinterpret_cast<const float4*>(p + i));
            f[i] = t.x; f[i + 1] = t.y; f[i + 2] = t.z; f[i + 3] = t.w;
        }
    }
}

template <int kBytes>
__device__ __forceinline__ void copy_async(uint32_t dst, const void* src) {
    if constexpr (kBytes == 32) {
        copy_async<16>(dst, src);
        copy_async<16>(dst + 16, static_cast<const char*>(src) + 16);
    } else if constexpr (kBytes == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(kBytes) : "memory");
}

__device__ __forceinline__ size_t tiled_index_offset(uint32_t m, uint32_t cb, uint32_t CB, uint32_t n_stile,
                                                     uint32_t cb_mtile) {
    // index_calc_host.cpp:41-49
    uint32_t n_tile = m / n_stile, n_in = m % n_stile;
    uint32_t cb_tile = cb / cb_mtile, cb_in = cb % cb_mtile;
    return (size_t)n_tile * n_stile * CB + (size_t)cb_tile * n_stile * cb_mtile + (size_t)n_in * cb_mtile + cb_in;
}

// Programmatic dependent launch, both kernels: launch_dependents at entry lets the LUT kernel queued behind
// start its prologue while the search runs (it waits for this grid before it reads the indices).  The kernel
// is itself a programmatic dependent of whatever precedes it: it stages its centroids - weights, which no
// preceding kernel writes - before griddepcontrol.wait, and touches activations and the index buffer, which
// the previous LUT kernel may still be reading, only after it.
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ------------------------------------------------------------------ thread <-> codebook
constexpr int kRegThreads = 128;

// The CTA takes W codebooks, one per thread, and its kRegThreads / W groups of threads different runs of tokens: they share
// one staged copy of the centroids.
// SHORT (W = 32): a thread takes one batch of kTok tokens and no more, the activations load straight into registers, and
// the scan runs as it is: a batch small enough for this is bound by a chain of latencies, which the filter would lengthen
// (0.3 us of a 15 us call).  Otherwise every thread takes a run of tokens.
//
// With 64 numbers a codebook registers hold the centroids for two tokens at a time, where ccs_tile_kernel reads them from
// shared memory.  Search alone, us, that kernel -> this one, N(0,1) and every centroid twice (all pairs undecided):
//     v = 4, 16 centroids   16384 x 768 codebooks   90 -> 72   256 -> 158        8192 x 256    21 -> 18    51 -> 33
//     v = 2, 32             4096 x 384              25 -> 17    68 -> 31         2000 x 1280   34 -> 24    96 -> 46
//     v = 8, 8              8192 x 1280             85 -> 62   191 -> 132        8192 x 384    33 -> 23    66 -> 44
// Both tokens have a margin of their own: with one for both, from the sum of their norms, half again as many pairs went to the scan
// (16384 x 768, v = 4, 16 centroids, an offset of 30: 242 us, 140 now, ccs_tile_kernel 218).  Four tokens share one, which saves
// what it costs.  The scan takes the centroids from the registers, two at a time; with single ones from shared memory,
// 12608 x 384, v = 2, 16 centroids that come twice took 76 us, 44 like this (and N(0,1) 26.0, 25.0).
template <int V, int CT, bool TILED, int kTok, bool SHORT, int W>
__global__ void __launch_bounds__(kRegThreads, SHORT ? (CT * V >= 64 ? 6 : 8) : CT * V >= 64 ? (CT == 32 ? 3 : 4) : CT * V >= 32 ? 5 : 7)
ccs_reg_kernel(const float* __restrict__ x, const float* __restrict__ cent, void* __restrict__ out, uint32_t M,
               uint32_t K, uint32_t CB, uint32_t tokens_per_cta, uint32_t n_stile, uint32_t cb_mtile) {
    pdl_launch();
    // tokens_per_cta is the run of ONE thread: the CTA's run, or each warp's where the warps take different tokens
    constexpr uint32_t kCbCta = W, kTokWarps = (uint32_t)kRegThreads / W;
    const uint32_t col = kTokWarps > 1 ? threadIdx.x % W : threadIdx.x;   // codebook of the CTA this thread works on
    const uint32_t cb = blockIdx.x * kCbCta + col;
    const uint32_t m0 = (blockIdx.y * kTokWarps + (kTokWarps > 1 ? threadIdx.x / W : 0u)) * tokens_per_cta;
    const uint32_t m1 = min(M, m0 + tokens_per_cta);
    const bool active = cb < CB && m0 < M;

    const float* xp = x + (size_t)(active ? cb : 0) * V;
    // Activations arrive through a ring of kRing batches of kTok tokens in shared memory, every thread copying and
    // reading its own bytes only (no barrier): 12 rows ahead instead of the 4 that registers have room for.  With
    // 4, the copies in flight (17 KB per SM) held a 12608 x 3072 search to 1.9 TB/s, its first stall reason.
    constexpr int kRing = SHORT ? 1 : V == 2 ? 4 : 3;
    __shared__ __align__(16) float s_ring[kRing][kTok][kRegThreads][V];
    const uint32_t ring0 = static_cast<uint32_t>(__cvta_generic_to_shared(&s_ring[0][0][threadIdx.x][0]));
    auto fetch = [&](uint32_t m, uint32_t slot) {   // rows past the end repeat the last one (their results are not stored)
        const uint32_t dst = ring0 + slot * (uint32_t)sizeof(s_ring[0]);
        if (m + kTok <= m1) {
            const float* p = xp + (size_t)m * K;
#pragma unroll
            for (int t = 0; t < kTok; ++t, p += K) copy_async<V * 4>(dst + t * (uint32_t)sizeof(s_ring[0][0]), p);
        } else if (m < m1) {
#pragma unroll
            for (int t = 0; t < kTok; ++t)
                copy_async<V * 4>(dst + t * (uint32_t)sizeof(s_ring[0][0]), xp + (size_t)min(m + t, M - 1) * K);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    // The CTA's codebooks are contiguous in memory: fetch them coalesced into shared memory, negated.  The row pitch
    // keeps the per-thread reads - a word at a time, or a vector in the SHORT form - free of bank conflicts.
    constexpr int kVec = SHORT ? (V == 2 ? 2 : 4) : 1;
    constexpr int kRow = CT * V, kPitch = kRow + kVec;
    __shared__ __align__(16) float s_cent[kCbCta * kPitch];
    {
        const uint32_t cb0 = blockIdx.x * kCbCta;
        const uint32_t n_cb = min(kCbCta, CB - cb0);
        const float* gp = cent + (size_t)cb0 * kRow;
        for (uint32_t e = threadIdx.x; e < n_cb * kRow; e += kRegThreads) {
            const uint32_t r = e / kRow, i = e % kRow;
            s_cent[r * kPitch + i] = -__ldg(gp + e);
        }
    }
    pdl_wait();
    float cur[kTok][V];
    if constexpr (SHORT) {
#pragma unroll
        for (int t = 0; t < kTok; ++t) load_global<V>(xp + (size_t)min(m0 + t, M - 1) * K, cur[t]);
    } else {
#pragma unroll
        for (uint32_t r = 0; r + 1 < kRing; ++r) fetch(active ? m0 + r * kTok : m1, r);
    }
    __syncthreads();
    if (!active) return;

    const float* my_cent = s_cent + col * kPitch;
    auto store = [&](uint32_t m, const uint32_t (&best)[kTok]) {
        if constexpr (TILED) {
#pragma unroll
            for (int t = 0; t < kTok; ++t)
                if (m + t < m1) reinterpret_cast<uint16_t*>(out)[tiled_index_offset(m + t, cb, CB, n_stile, cb_mtile)] = (uint16_t)best[t];
        } else {
            uint8_t* o = reinterpret_cast<uint8_t*>(out) + (size_t)m * CB + cb;
            if (m + kTok <= m1) {
#pragma unroll
                for (int t = 0; t < kTok; ++t, o += CB) *o = (uint8_t)best[t];
            } else {
#pragma unroll
                for (int t = 0; t < kTok; ++t, o += CB)
                    if (m + t < m1) *o = (uint8_t)best[t];
            }
        }
    };
    if constexpr (SHORT) {
        float mn[kTok];
        uint32_t best[kTok];
#pragma unroll
        for (int c = 0; c < CT; ++c) {
            float nc[V];
            load_x<V>(my_cent + c * V, nc);
#pragma unroll
            for (int t = 0; t < kTok; ++t) {
                // two components per packed instruction; each lane of it rounds on its own, and the addition and
                // the multiplication stay separate instructions
                float acc = 0.f;
#pragma unroll
                for (int d = 0; d < V; d += 2) {
                    const float2 e = __fadd2_rn(make_float2(cur[t][d], cur[t][d + 1]), make_float2(nc[d], nc[d + 1]));
                    const float2 sq = __fmul2_rn(e, e);
                    acc = d == 0 ? sq.x : __fadd_rn(acc, sq.x);  // 0 + sq.x is exact
                    acc = __fadd_rn(acc, sq.y);
                }
                const bool take = c == 0 || __fsub_rn(mn[t], acc) > kEps;  // false for NaN: keeps the earlier index
                mn[t] = take ? acc : mn[t];
                best[t] = take ? (uint32_t)c : best[t];
            }
        }
        store(m0, best);
        return;
    } else {
        float2 nc[CT / 2][V], h[CT / 2];   // two centroids per pair: one packed instruction works on both
        float t_cb = kMarginBase;
        {
            float top = 0.f;
            bool fine = true;
#pragma unroll
            for (int j = 0; j < CT / 2; ++j) {
                float2 cc = make_float2(0.f, 0.f);
#pragma unroll
                for (int d = 0; d < V; ++d) {
                    nc[j][d] = make_float2(my_cent[2 * j * V + d], my_cent[(2 * j + 1) * V + d]);
                    cc = __ffma2_rn(nc[j][d], nc[j][d], cc);
                }
                h[j] = make_float2(0.5f * cc.x, 0.5f * cc.y);
                fine = fine && cc.x < kHuge && cc.y < kHuge;
                top = fmaxf(top, fmaxf(cc.x, cc.y));
            }
            t_cb = fine ? fmaf(margin_factor(V), top, kMarginBase) : __int_as_float(0x7f800000);
        }

        // The reference's scan, two centroids at a time from the registers that hold them.
        auto scan = [&](const float (&x)[V]) {
            float mn = 0.f;
            uint32_t best = 0;
#pragma unroll
            for (int j = 0; j < CT / 2; ++j) {
                float2 acc = make_float2(0.f, 0.f);
#pragma unroll
                for (int d = 0; d < V; ++d) {
                    const float2 e = __fadd2_rn(make_float2(x[d], x[d]), nc[j][d]);
                    const float2 sq = __fmul2_rn(e, e);
                    // 0 + sq is exact.  Scalar additions: a packed one is contracted with the packed multiplication
                    acc = d == 0 ? sq : make_float2(__fadd_rn(acc.x, sq.x), __fadd_rn(acc.y, sq.y));
                }
                const bool take = j == 0 || __fsub_rn(mn, acc.x) > kEps;  // false for NaN: keeps the earlier index
                mn = take ? acc.x : mn;
                best = take ? (uint32_t)(2 * j) : best;
                const bool next = __fsub_rn(mn, acc.y) > kEps;
                mn = next ? acc.y : mn;
                best = next ? (uint32_t)(2 * j + 1) : best;
            }
            return best;
        };
        auto search = [&](uint32_t m) {
            // one margin for the kTok tokens: that of the sum of their norms.  Of two, each has its own
            constexpr int kMargins = kTok == 2 ? 2 : 1;
            float2 xx[kMargins] = {};
#pragma unroll
            for (int t = 0; t < kTok; ++t)
#pragma unroll
                for (int d = 0; d < V; d += 2) {
                    const float2 q = make_float2(cur[t][d], cur[t][d + 1]);
                    xx[t % kMargins] = __ffma2_rn(q, q, xx[t % kMargins]);
                }
            float T[kTok];
            bool sound = true;
#pragma unroll
            for (int t = 0; t < kTok; ++t) {
                T[t] = fmaf(margin_factor(V), xx[t % kMargins].x + xx[t % kMargins].y, t_cb);
                sound = sound && T[t] < kHuge;
            }
            uint32_t mask[kTok], best[kTok], several = 0;
#pragma unroll
            for (int t = 0; t < kTok; ++t) {
                float k[CT];
#pragma unroll
                for (int j = 0; j < CT / 2; ++j) {
                    float2 s = h[j];
#pragma unroll
                    for (int d = 0; d < V; ++d) s = __ffma2_rn(make_float2(cur[t][d], cur[t][d]), nc[j][d], s);
                    k[2 * j] = s.x;
                    k[2 * j + 1] = s.y;
                }
                mask[t] = below<CT>(k, min_of(k) + T[t]);
                best[t] = high_bit(mask[t]);
                several |= all_but_lowest(mask[t]);
            }
            if (several != 0 || !sound) {
#pragma unroll
                for (int t = 0; t < kTok; ++t)
                    if (!(T[t] < kHuge) || all_but_lowest(mask[t]) != 0) best[t] = scan(cur[t]);
            }
            store(m, best);
        };
        uint32_t slot = 0, ahead = kRing - 1;
        for (uint32_t m = m0; m < m1; m += kTok) {
            asm volatile("cp.async.wait_group %0;" ::"n"(SHORT ? 0 : kRing - 2) : "memory");
#pragma unroll
            for (int t = 0; t < kTok; ++t) load_x<V>(&s_ring[slot][t][threadIdx.x][0], cur[t]);
            fetch(m + (kRing - 1) * kTok, ahead);
            if (++slot == kRing) slot = 0;
            if (++ahead == kRing) ahead = 0;
            search(m);
        }
    }
}

// ------------------------------------------------------------------ thread <-> token
constexpr int kTileThreads = 128;

// codebooks of one CTA: about 128 to 192 bytes of a token's row
__host__ __device__ constexpr int tile_codebooks(int v) {
    return v == 1 ? 16 : v == 2 ? 8 : v <= 12 ? 4 : v <= 24 ? 2 : 1;
}
// Row pitch of the staged activations, in floats: 4 mod 8 keeps 16-byte copies aligned and 16-byte reads of 32 rows
// free of bank conflicts; odd lengths are read word by word, which an odd pitch serves.
__host__ __device__ constexpr int tile_pitch(int v) {
    const int w = tile_codebooks(v) * v;
    return v % 2 ? (w | 1) : (w + 3) / 8 * 8 + 4;
}
// From 12 components on, packed instructions take two components of one centroid (one horizontal addition per
// key); below, two centroids (the activations are duplicated into register pairs, which long vectors cannot afford).
__host__ __device__ constexpr bool tile_pairs_components(int v) { return v >= 12 && v % 4 == 0; }

// Where component d of centroid c of a codebook lies in its staged block: quads of centroids, V + 1 groups of four
// floats each.  Pairs of centroids: group d holds component d of the four, group V their |c|^2 / 2.  Pairs of
// components: the four centroids one after the other, then their |c|^2 / 2.
template <int V>
__device__ __forceinline__ uint32_t cent_at(uint32_t c, uint32_t d) {
    const uint32_t quad = (c >> 2) * (4 * (V + 1)), in = c & 3u;
    if constexpr (tile_pairs_components(V)) return quad + in * V + d;
    else return quad + d * 4 + in;
}

// G: centroids whose keys are held at once.  ONE: num_centroid <= G, so there is a single group.
template <int V, int G, bool ONE, int kTok, bool TILED>
__global__ void __launch_bounds__(kTileThreads, V <= 5 ? 6 : 4)
ccs_tile_kernel(const float* __restrict__ x, const float* __restrict__ cent, void* __restrict__ out, uint32_t M,
                uint32_t K, uint32_t CB, uint32_t CT, uint32_t copy16, uint32_t words, uint32_t n_stile, uint32_t cb_mtile) {
    constexpr int kCbs = tile_codebooks(V), kPitch = tile_pitch(V), kTokens = kTileThreads * kTok;
    constexpr bool kPairD = tile_pairs_components(V);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    pdl_launch();
    float* s_x = reinterpret_cast<float*>(smem_raw);                    // [kTokens][kPitch]
    constexpr int kXFloats = (kTokens * kPitch + 3) / 4 * 4;
    float* s_c = s_x + kXFloats;                                        // [kCbs][groups][G/4][V+1][4]
    __shared__ uint32_t s_top[kCbs];                                    // max |c|^2 as bits (NaN and infinity sort last)
    const uint32_t groups = ONE ? 1u : (CT + G - 1) / G, ct_pad = groups * G;
    const uint32_t c_block = ct_pad * (V + 1);
    const uint32_t cb0 = blockIdx.x * kCbs, cbs = min((uint32_t)kCbs, CB - cb0);
    const uint32_t m_base = blockIdx.y * kTokens;

    if (threadIdx.x < kCbs) s_top[threadIdx.x] = 0;
    __syncthreads();
    for (uint32_t e = threadIdx.x; e < cbs * ct_pad; e += kTileThreads) {
        const uint32_t b = e / ct_pad, c = e % ct_pad;
        float v[V], cc = 0.f;
        if (c < CT) {
            const float* g = cent + ((size_t)(cb0 + b) * CT + c) * V;
#pragma unroll
            for (int d = 0; d < V; ++d) v[d] = -__ldg(g + d);
        } else {
#pragma unroll
            for (int d = 0; d < V; ++d) v[d] = 0.f;
        }
#pragma unroll
        for (int d = 0; d < V; ++d) cc = fmaf(v[d], v[d], cc);
        float* blk = s_c + b * c_block;
#pragma unroll
        for (int d = 0; d < V; ++d) blk[cent_at<V>(c, d)] = v[d];
        blk[(c >> 2) * (4 * (V + 1)) + 4 * V + (c & 3u)] = c < CT ? 0.5f * cc : __int_as_float(0x7f800000);
        atomicMax(&s_top[b], __float_as_uint(cc));
    }
    pdl_wait();
    {
        const float* xg = x + (size_t)cb0 * V;
        const uint32_t rows = min((uint32_t)kTokens, M - m_base);
        const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(s_x));
        constexpr uint32_t kW = kCbs * V;
        const uint32_t w = cbs * V;
        if (V % 2 == 0 && kW % 4 == 0 && copy16) {
            // A thread keeps its column of 16 bytes and walks down the rows, so that a copy costs two additions.  With a
            // division per copy a warp and codebook took 298 instructions at v = 10, 16 centroids; 250 like this: 8192 x 1024
            // 137 -> 122 us with its contraction (v = 20 138 -> 123, v = 8 131 -> 125).
            constexpr uint32_t kQ = kW / 4, kRows = kTileThreads / kQ;   // rows of one turn
            const uint32_t q = threadIdx.x % kQ;
            uint32_t r = threadIdx.x / kQ, to = dst + (r * kPitch + 4 * q) * 4;
            if (r < kRows && 4 * q < w) {
                const float* from = xg + (size_t)(m_base + r) * K + 4 * q;
                const size_t step = (size_t)kRows * K;
#pragma unroll 4
                for (; r < rows; r += kRows, to += kRows * kPitch * 4, from += step) copy_async<16>(to, from);
            }
        } else {
            for (uint32_t i = threadIdx.x; i < rows * kW; i += kTileThreads) {
                const uint32_t r = i / kW, q = i % kW;
                if (q < w) copy_async<4>(dst + (r * kPitch + q) * 4, xg + (size_t)(m_base + r) * K + q);
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    __syncthreads();

    uint32_t word[kTok] = {};
#pragma unroll 1
    for (uint32_t b = 0; b < cbs; ++b) {
        const float* blk = s_c + b * c_block;
        float xv[kTok][V], T[kTok], m1[kTok];
        uint32_t cand[kTok], base[kTok];
        {
            const float top = __uint_as_float(s_top[b]);
            const float t_cb = top < kHuge ? fmaf(margin_factor(V), top, kMarginBase) : __int_as_float(0x7f800000);
#pragma unroll
            for (int t = 0; t < kTok; ++t) {
                const float* row = s_x + (threadIdx.x + t * kTileThreads) * kPitch + b * V;
                float xx = 0.f;
                load_x<V>(row, xv[t]);
#pragma unroll
                for (int d = 0; d < V; ++d) xx = fmaf(xv[t][d], xv[t][d], xx);
                T[t] = fmaf(margin_factor(V), xx, t_cb);
                m1[t] = __int_as_float(0x7f800000);
                cand[t] = 0;
                base[t] = 0;
            }
        }
#pragma unroll 1
        for (uint32_t g = 0; g < groups; ++g) {
            float k[kTok][G];
            const float* gp = blk + g * (G * (V + 1));
#pragma unroll
            for (int q = 0; q < G / 4; ++q) {
                const float* qp = gp + q * (4 * (V + 1));
                const float4 h = *reinterpret_cast<const float4*>(qp + 4 * V);
                if constexpr (kPairD) {
                    const float hs[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        float2 s[kTok];
#pragma unroll
                        for (int t = 0; t < kTok; ++t) s[t] = make_float2(hs[c], 0.f);
#pragma unroll
                        for (int d = 0; d < V; d += 4) {
                            const float4 cv = *reinterpret_cast<const float4*>(qp + c * V + d);
#pragma unroll
                            for (int t = 0; t < kTok; ++t) {
                                s[t] = __ffma2_rn(make_float2(xv[t][d], xv[t][d + 1]), make_float2(cv.x, cv.y), s[t]);
                                s[t] = __ffma2_rn(make_float2(xv[t][d + 2], xv[t][d + 3]), make_float2(cv.z, cv.w), s[t]);
                            }
                        }
#pragma unroll
                        for (int t = 0; t < kTok; ++t) k[t][4 * q + c] = s[t].x + s[t].y;
                    }
                } else {
                    float2 lo[kTok], hi[kTok];
#pragma unroll
                    for (int t = 0; t < kTok; ++t) { lo[t] = make_float2(h.x, h.y); hi[t] = make_float2(h.z, h.w); }
#pragma unroll
                    for (int d = 0; d < V; ++d) {
                        const float4 cv = *reinterpret_cast<const float4*>(qp + 4 * d);
#pragma unroll
                        for (int t = 0; t < kTok; ++t) {
                            const float2 xd = make_float2(xv[t][d], xv[t][d]);
                            lo[t] = __ffma2_rn(xd, make_float2(cv.x, cv.y), lo[t]);
                            hi[t] = __ffma2_rn(xd, make_float2(cv.z, cv.w), hi[t]);
                        }
                    }
#pragma unroll
                    for (int t = 0; t < kTok; ++t) {
                        k[t][4 * q] = lo[t].x; k[t][4 * q + 1] = lo[t].y; k[t][4 * q + 2] = hi[t].x; k[t][4 * q + 3] = hi[t].y;
                    }
                }
            }
#pragma unroll
            for (int t = 0; t < kTok; ++t) {
                const float gm = min_of(k[t]);
                if constexpr (ONE) {
                    cand[t] = below<G>(k[t], gm + T[t]);
                } else {
                    // Candidates so far survive if the smallest of them is still within the margin; together with
                    // new ones they are more than one.
                    const float now = fminf(m1[t], gm), thr = now + T[t];
                    const uint32_t mask = below<G>(k[t], thr);
                    const bool keep = m1[t] < thr;
                    if (mask) {
                        cand[t] = keep ? 0xFFFFFFFFu : mask;
                        base[t] = g * G;
                    }
                    m1[t] = now;
                }
            }
        }
#pragma unroll
        for (int t = 0; t < kTok; ++t) {
            uint32_t best = base[t] + high_bit(cand[t]);
            const uint32_t m = m_base + threadIdx.x + t * kTileThreads;
            if (m < M && (!(T[t] < kHuge) || all_but_lowest(cand[t]) != 0))
                best = exact_scan<V>(xv[t], CT, [&](uint32_t c, int d) { return blk[cent_at<V>(c, d)]; });
            if constexpr (TILED) {
                if (m < M) reinterpret_cast<uint16_t*>(out)[tiled_index_offset(m, cb0 + b, CB, n_stile, cb_mtile)] = (uint16_t)best;
            } else {
                uint8_t* o = reinterpret_cast<uint8_t*>(out) + (size_t)m * CB + cb0;
                if (kCbs % 4 == 0 && words) {   // four codebooks per store
                    word[t] |= best << (8 * (b & 3u));
                    if ((b & 3u) == 3u) {
                        if (m < M) *reinterpret_cast<uint32_t*>(o + (b & ~3u)) = word[t];
                        word[t] = 0;
                    }
                } else if (m < M) {
                    o[b] = (uint8_t)best;
                }
            }
        }
    }
}

// ------------------------------------------------------------------ any sub-vector length
constexpr int kAnyThreads = 128;  // tokens per CTA

// Run-time length: thread <-> token, centroids of a block of codebooks in shared memory, the token's slice is
// re-read (L1 resident) per centroid; exact_scan's arithmetic without the filter.
template <bool TILED>
__global__ void __launch_bounds__(kAnyThreads)
ccs_any_kernel(const float* __restrict__ x, const float* __restrict__ cent, void* __restrict__ out, uint32_t M,
               uint32_t K, uint32_t v, uint32_t CB, uint32_t CT, uint32_t cb_per_cta, uint32_t n_stile,
               uint32_t cb_mtile) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    pdl_launch();
    pdl_wait();
    float* s_cent = reinterpret_cast<float*>(smem_raw);                   // [cbs][CT][v]
    const uint32_t cb0 = blockIdx.x * cb_per_cta;
    const uint32_t cbs = min(cb_per_cta, CB - cb0);
    uint8_t* s_idx = smem_raw + (size_t)cb_per_cta * CT * v * sizeof(float);  // [128][cb_per_cta]

    const uint32_t n_c = cbs * CT * v;
    const float* gc = cent + (size_t)cb0 * CT * v;
    for (uint32_t i = threadIdx.x; i < n_c; i += kAnyThreads) s_cent[i] = __ldg(gc + i);
    __syncthreads();

    const uint32_t m_base = blockIdx.y * kAnyThreads;
    const uint32_t m = m_base + threadIdx.x;
    if (m < M) {
        const float* xp = x + (size_t)m * K + (size_t)cb0 * v;
        for (uint32_t cl = 0; cl < cbs; ++cl, xp += v) {
            const float* cp = s_cent + (size_t)cl * CT * v;
            float mn = 0.f;
            uint32_t best = 0;
            for (uint32_t ct = 0; ct < CT; ++ct) {
                float t = 0.f;
                for (uint32_t d = 0; d < v; ++d) {
                    float e = __fsub_rn(__ldg(xp + d), cp[ct * v + d]);
                    t = __fadd_rn(t, __fmul_rn(e, e));
                }
                bool take = (ct > 0) && (__fsub_rn(mn, t) > kEps);
                if (ct == 0) mn = t;
                mn = take ? t : mn;
                best = take ? ct : best;
            }
            s_idx[threadIdx.x * cb_per_cta + cl] = (uint8_t)best;
        }
    }
    __syncthreads();
    // write-out: consecutive threads -> consecutive codebooks of one token
    const uint32_t rows = min((uint32_t)kAnyThreads, M > m_base ? M - m_base : 0u);
    for (uint32_t i = threadIdx.x; i < rows * cbs; i += kAnyThreads) {
        uint32_t r = i / cbs, cl = i % cbs;
        uint8_t b = s_idx[r * cb_per_cta + cl];
        if constexpr (TILED) {
            reinterpret_cast<uint16_t*>(out)[tiled_index_offset(m_base + r, cb0 + cl, CB, n_stile, cb_mtile)] = b;
        } else {
            reinterpret_cast<uint8_t*>(out)[(size_t)(m_base + r) * CB + cb0 + cl] = b;
        }
    }
}

// Launch with programmatic stream serialisation allowed: see pdl_wait.
template <typename... KArgs, typename... Args>
cudaError_t launch_dependent(void (*k)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, static_cast<KArgs>(args)...);
}

// Number of SMs of the current device (the same for every device of one kind)
uint32_t sm_count() {
    static const uint32_t n = [] {
        int dev = 0, v = 0;
        cudaGetDevice(&dev);
        return cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && v > 0 ? (uint32_t)v : 148u;
    }();
    return n;
}

template <int V, int CT, int kTok, bool SHORT, int W>
uint32_t resident_ctas() {
    static const uint32_t n = [] {
        int r = 0;
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, ccs_reg_kernel<V, CT, false, kTok, SHORT, W>, kRegThreads, 0) == cudaSuccess && r > 0 ? (uint32_t)r : 4u;
    }();
    return n * sm_count();
}

template <int V, int CT, int kTok, bool SHORT, int W>
cudaError_t run_reg_grid(const CcsArgs& a, dim3 grid, uint32_t run, cudaStream_t s) {
    auto k = a.format == LUTAMM_INDEX_U16_TILED ? ccs_reg_kernel<V, CT, true, kTok, SHORT, W> : ccs_reg_kernel<V, CT, false, kTok, SHORT, W>;
    return launch_dependent(k, grid, dim3(kRegThreads), 0, s, a.x, a.centroid, a.idx_out, a.M, a.K, a.CB, run, a.n_stile, a.cb_mtile);
}

constexpr uint64_t kMostGridY = 65535, kLongestRun = 192;
constexpr uint32_t kTok = 4;   // tokens whose activations a thread loads together: one round trip to memory instead of four

// tokens of a batch in a run: two where the centroids leave no registers, and no shared memory, for four
constexpr int run_tok(int v, int CT) { return v * CT >= 64 ? 2 : (int)kTok; }

// One batch of kTok tokens per thread, while the GPU holds all those CTAs at once.
template <int V, int CT>
bool short_fits(const CcsArgs& a, dim3* grid) {
    *grid = dim3((a.CB + 31) / 32, (a.M + 4 * kTok - 1) / (4 * kTok));
    return !a.tokens_per_thread && (uint64_t)grid->x * grid->y <= resident_ctas<V, CT, kTok, true, 32>();
}

template <int V, int CT, int W>
cudaError_t run_reg_width(const CcsArgs& a, cudaStream_t s) {
    constexpr int kTok = run_tok(V, CT);
    constexpr uint64_t kGroups = kRegThreads / W;   // of threads that take different runs
    const uint64_t cb_blocks = (a.CB + W - 1) / W;
    uint64_t run = a.tokens_per_thread;
    if (!run) {
        // Waves of equal runs of up to 192 tokens, filled as far as whole runs fill them: a last wave that is a third full
        // costs as much as a full one, and staging the centroids costs a few microseconds per wave (32 tokens' worth).
        // In longer runs CTAs that read the same rows drift apart (65536 x 784 codebooks, v = 2, 32 centroids: a wave of 964 tokens
        // 351 us, 384 tokens 365, 96 to 256 335 to 343; v = 4, 16 centroids: a wave of 712 273, 384 285, 96 to 256 256 to 264).  A cap of
        // 128 or 256 does the same within 1 % on average over 140 calls.
        const uint64_t wave = resident_ctas<V, CT, kTok, false, W>(), cap = kLongestRun * kGroups;
        const uint64_t fewest = (cb_blocks * ((a.M + cap - 1) / cap) + wave - 1) / wave;
        uint64_t least = ~0ull;
        for (uint64_t waves = fewest; waves < fewest + 4; ++waves) {
            const uint64_t rows = waves * wave / cb_blocks;   // CTAs of a block of codebooks
            if (!rows) continue;
            const uint64_t r = (a.M + rows * kGroups - 1) / (rows * kGroups), cost = waves * (r + 32);
            if (cost < least) { least = cost; run = r; }
        }
        if (!run) run = kLongestRun;
    }
    // what a plan names, as far as the grid holds it and there are tokens (a run of 2^32 - 1 rounds up to none)
    run = std::clamp(run, (a.M + kMostGridY * kGroups - 1) / (kMostGridY * kGroups), (a.M + kGroups - 1) / kGroups);
    const uint32_t tokens = (uint32_t)((run + kTok - 1) / kTok * kTok);
    return run_reg_grid<V, CT, kTok, false, W>(a, dim3((uint32_t)cb_blocks, (uint32_t)((a.M + tokens * kGroups - 1) / (tokens * kGroups))), tokens, s);
}

template <int V, int CT>
cudaError_t run_reg(const CcsArgs& a, cudaStream_t s) {
    // Search alone, us, blocks of 32 codebooks and of 128.  Narrow ones waste fewer threads (32768 x 192, v = 4, 16 centroids 39
    // and 51) and make shorter waves (8192 x 256 18.0 and 18.6; 1576 x 1024, v = 2 12.8 and 13.1).  Wide ones read 1 to 2 KB of a row
    // at once, which pays where wide rows come from memory throughout (32768 x 1024, v = 4 177 and 169; 20000 x 1536 163 and 157).
    // (at v = 8 a narrow block reads 1 KB, and the wide one's centroids and batches are more shared memory than there is)
    if constexpr (V == 8) return run_reg_width<V, CT, 32>(a, s);
    else return a.M >= 10000 && a.CB >= 768 && a.CB % 128 == 0 ? run_reg_width<V, CT, 128>(a, s) : run_reg_width<V, CT, 32>(a, s);
}

template <int V, int G, bool ONE, int kTok>
cudaError_t run_tile_tok(const CcsArgs& a, size_t smem, cudaStream_t s) {
    constexpr uint32_t kCbs = tile_codebooks(V);
    const uint32_t tokens = kTileThreads * kTok;
    const dim3 grid((a.CB + kCbs - 1) / kCbs, (a.M + tokens - 1) / tokens);
    if (grid.y > 65535u) return cudaErrorInvalidValue;
    const uint32_t copy16 = a.K % 4 == 0 && reinterpret_cast<uintptr_t>(a.x) % 16 == 0;
    const uint32_t words = a.CB % 4 == 0 && reinterpret_cast<uintptr_t>(a.idx_out) % 4 == 0;
    auto k = a.format == LUTAMM_INDEX_U16_TILED ? ccs_tile_kernel<V, G, ONE, kTok, true> : ccs_tile_kernel<V, G, ONE, kTok, false>;
    static SmemOptIn memo[2];
    cudaError_t e = allow_smem(memo[a.format == LUTAMM_INDEX_U16_TILED], k, (int)smem);
    if (e != cudaSuccess) return e;
    return launch_dependent(k, grid, dim3(kTileThreads), smem, s, a.x, a.centroid, a.idx_out, a.M, a.K, a.CB, a.CT, copy16, words,
                            a.n_stile, a.cb_mtile);
}

template <int V>
cudaError_t run_tile(const CcsArgs& a, cudaStream_t s) {
    constexpr uint32_t kCbs = tile_codebooks(V);
    const uint32_t g = a.CT <= 8 ? 8 : 16, ct_pad = (a.CT + g - 1) / g * g;
    auto smem = [&](uint32_t tok) { return ((size_t)(kTileThreads * tok * tile_pitch(V) + 3) / 4 * 4 + (size_t)kCbs * ct_pad * (V + 1)) * sizeof(float); };
    // Two tokens per thread share each centroid read; one where that would leave SMs without a CTA.
    const uint64_t ctas2 = (uint64_t)((a.CB + kCbs - 1) / kCbs) * ((a.M + 2 * kTileThreads - 1) / (2 * kTileThreads));
    const bool two = ctas2 >= 2ull * sm_count() && smem(2) <= 112 * 1024;
    if (g == 8) return two ? run_tile_tok<V, 8, true, 2>(a, smem(2), s) : run_tile_tok<V, 8, true, 1>(a, smem(1), s);
    if (a.CT <= 16) return two ? run_tile_tok<V, 16, true, 2>(a, smem(2), s) : run_tile_tok<V, 16, true, 1>(a, smem(1), s);
    return two ? run_tile_tok<V, 16, false, 2>(a, smem(2), s) : run_tile_tok<V, 16, false, 1>(a, smem(1), s);
}

cudaError_t run_any(const CcsArgs& a, cudaStream_t s) {
    // centroid tile + index tile per CTA; keep under ~96 KB so two CTAs fit an SM
    const size_t per_cb = (size_t)a.CT * a.v * sizeof(float) + kAnyThreads;
    uint32_t cb_per_cta = (uint32_t)((96 * 1024) / per_cb);
    if (cb_per_cta == 0) cb_per_cta = 1;
    if (cb_per_cta > 64) cb_per_cta = 64;
    if (cb_per_cta > a.CB) cb_per_cta = a.CB;
    const size_t smem = per_cb * cb_per_cta;
    if (smem > 200 * 1024) return cudaErrorInvalidValue;
    dim3 grid((a.CB + cb_per_cta - 1) / cb_per_cta, (a.M + kAnyThreads - 1) / kAnyThreads);
    auto k = a.format == LUTAMM_INDEX_U16_TILED ? ccs_any_kernel<true> : ccs_any_kernel<false>;
    static SmemOptIn memo[2];
    cudaError_t e = allow_smem(memo[a.format == LUTAMM_INDEX_U16_TILED], k, (int)smem);
    if (e != cudaSuccess) return e;
    return launch_dependent(k, grid, dim3(kAnyThreads), smem, s, a.x, a.centroid, a.idx_out, a.M, a.K, a.v, a.CB, a.CT,
                            cb_per_cta, a.n_stile, a.cb_mtile);
}

// The instances with a short form, and those whose thread walks a run of tokens.
#define LUTAMM_CCS_SHORT_INSTANCES(X) X(2, 8) X(2, 16) X(2, 32) X(4, 8) X(4, 16) X(8, 8) X(8, 16)
#define LUTAMM_CCS_RUN_INSTANCES(X) X(2, 8) X(2, 16) X(4, 8) X(4, 16) X(2, 32) X(8, 8)

}  // namespace

// Whether tokens_per_thread changes anything but the choice of the short form.
bool ccs_reads_tokens_per_thread(uint32_t v, uint32_t CT) {
#define LUTAMM_CCS_IS(V_, CT_) || (v == V_ && CT == CT_)
    return false LUTAMM_CCS_RUN_INSTANCES(LUTAMM_CCS_IS);
}
bool ccs_has_short_form(uint32_t v, uint32_t CT) {
    return false LUTAMM_CCS_SHORT_INSTANCES(LUTAMM_CCS_IS);
}
uint32_t ccs_light_ctas(uint32_t M, uint32_t CB, uint32_t CT, uint32_t v) {
    const uint64_t ctas = (uint64_t)((CB + 31) / 32) * ((M + 4 * kTok - 1) / (4 * kTok));
    return ccs_has_short_form(v, CT) && CT * v <= 64 && ctas < 1u << 30 ? (uint32_t)ctas : 0;
}
#undef LUTAMM_CCS_IS

cudaError_t launch_ccs(const CcsArgs& a, cudaStream_t s, const char** why) {
    *why = nullptr;
    if (a.M == 0 || a.CB == 0) return cudaSuccess;
    if (a.CT == 0 || a.CT > 256 || a.v == 0 || a.K != a.CB * a.v) {
        *why = "closest-centroid search: need 1 <= num_centroid <= 256 and input_feature_len == num_codebook*sub_vec_len";
        return cudaErrorInvalidValue;
    }
    if (ccs_umma_takes(a)) return launch_ccs_umma(a, s);
    // vector loads need the row pitch and the base address aligned to the vector width
    const uintptr_t xa = reinterpret_cast<uintptr_t>(a.x);
    const uint32_t vec_bytes = (a.v % 4 == 0) ? 16u : (a.v % 2 == 0) ? 8u : 4u;
    if (xa % vec_bytes == 0) {
        dim3 grid;
#define LUTAMM_CCS_SHORT(V_, CT_) \
    if (a.v == V_ && a.CT == CT_ && short_fits<V_, CT_>(a, &grid)) return run_reg_grid<V_, CT_, kTok, true, 32>(a, grid, kTok, s);
        LUTAMM_CCS_SHORT_INSTANCES(LUTAMM_CCS_SHORT)
#undef LUTAMM_CCS_SHORT
#define LUTAMM_CCS_REG(V_, CT_) \
    if (a.v == V_ && a.CT == CT_) return run_reg<V_, CT_>(a, s);
        LUTAMM_CCS_RUN_INSTANCES(LUTAMM_CCS_REG)
#undef LUTAMM_CCS_REG
    }
    switch (a.v) {
#define LUTAMM_CCS_TILE(V_) \
    case V_: return run_tile<V_>(a, s);
        LUTAMM_CCS_TILE(1)
        LUTAMM_CCS_TILE(2)
        LUTAMM_CCS_TILE(4)
        LUTAMM_CCS_TILE(8)
        LUTAMM_CCS_TILE(16)
        LUTAMM_CCS_TILE(32)
        // hidden sizes that are not a power of two times the codebook count (2560 / 256, 5120 / 256, ...)
        LUTAMM_CCS_TILE(3)
        LUTAMM_CCS_TILE(5)
        LUTAMM_CCS_TILE(6)
        LUTAMM_CCS_TILE(10)
        LUTAMM_CCS_TILE(12)
        LUTAMM_CCS_TILE(20)
        LUTAMM_CCS_TILE(24)
#undef LUTAMM_CCS_TILE
        default: return run_any(a, s);
    }
}

}  // namespace lutamm
