// Step 1 of the AMM on the tensor cores: the filter of ccs_argmin.cu with its scores s_c = |c|^2 / 2 - x.c from
// tcgen05.mma, for calls of many tokens.
//
// Replaces index_calculation() of the reference (inference-engine/src/host/index_calc_host.cpp:8-53), bit for bit like
// the other search kernels: a score only decides where it is certain, and every doubtful (token, codebook) goes on to the
// reference's scan (ccs_scan.cuh).
//
// Every component is split into two f16 numbers, a = hi + lo to 22 bits, and a codebook's contraction axis holds
//     activations   hi   hi   lo   1   1        centroids   -hi  -lo  -hi   hi(h)  lo(h)      h = |c|^2 / 2
// 3v + 2 positions rounded up to 16.  A CTA scales its activations and centroids by the power of two that brings the largest
// centroid component to 8..16, so nothing leaves f16's range that an ordinary table holds.  In scaled numbers, with
// A = |x|^2, B = max |c|^2 and u = 2^-24, |s computed - s| is at most
//     6u (A+B)             of the split (2^-22 of x, of c, and the missing lo.lo, on sum |x_d c_d| <= (A+B)/2), 3u B of h's,
//     (v+1) u B            of h itself,
//     2 (3v+4) u (A+B)     of the accumulation, each of the 3v+2 products off by a whole unit in the last place of the
//                          largest, twice (how the unit rounds is not documented),
//     17v 2^-25            where a component's lo is subnormal,
// so a margin of that twice and the fp32 filter's own, (22v + 54) u (A+B), would do; (24v + 64) is used, three times the
// fp32 filter's.  Measured against 64 bits the scores were off by at most 4 u (A+B) (v = 2, 4, 8 with 32 to 128 centroids:
// N(0,1), the same in thousandths, a hundred added, rows and centroids at mixed magnitudes).  The scores are 22-bit numbers
// where the other filter's are fp32; no score leaves the kernel, and no index depends on one that the margin does not settle.
// Rows with |x|^2 beyond 2^29 in scaled numbers, and what is not finite, take the scan.
//
// What bounds it: dispatch, like the other kernels.  Per centroid two instructions of selection and half a minimum are
// left, and nothing is read from shared memory; a token's codebook costs about 70 more (splitting, margin, hand-overs).
// The tensor pipe is 5 % busy.  Where ccs_reg_kernel has the centroids in registers the 70 outweigh what is saved (search and a
// 192-column contraction, that one and this one, us: 12608 x 1536, v = 2, 16 centroids 99 and 110; 32768 x 1536, v = 2, 32 433 and 452,
// 4096 x 768 43 and 48, 16384 x 384 61 and 64).
//
// The scan of undecided pairs is bound by the load/store unit (75 % busy where all are undecided): a centroid that all lanes
// read costs it as much as 32 different ones.  Undecided pairs wait in a queue of their warp, which holds all of a tile, and
// are scanned 32 at a time (scanned on the spot they held the other warps up).  Where more than three quarters of a tile's
// were undecided - centroids that come twice, a common offset large against their spread - the warp scans the next seven
// tiles without a look at the scores.  (A queue of candidates for the fp32 filter, 64 of them and the whole tile anew when
// there were more, took up to five times what ccs_tile_kernel takes.)
//
// Search and a 192-column contraction, us, ccs_tile_kernel -> this one, N(0,1) and every centroid twice:
//     32768 x 768 codebooks, v = 4, 64 centroids     583 -> 438     1961 -> 1456
//      8192 x 768, v = 4, 128                        304 -> 217      997 -> 689
//     32768 x 384, v = 8, 32                         262 -> 201      826 -> 760
//     16384 x 96, v = 8, 64                           72 -> 46       222 -> 168
//      8192 x 768, v = 4, 32                          91 -> 82       267 -> 218
//
// A CTA of four warps takes CC codebooks and a run of tiles of 128 tokens.  A tile is split into f16 in shared memory
// (K-major core matrices without swizzle, a pitch that spreads the stores over the banks) while the tile before is
// searched, from activations loaded one tile earlier still.  One thread issues the instructions of up to 128 columns; each
// thread reads the scores of one token back from tensor memory, 64 at a time, and the warp that reads last has the next
// columns computed.  No barrier in that loop: warps meet at these counts alone.  128 columns of tensor memory a CTA: four
// CTAs share an SM, and what one of them waits for the others hide (two buffers of 64 columns cost a hand-over per 64
// scores: 119 us where this took 102).
#include "kernels.h"
#include "ccs_scan.cuh"
#include "ptx.cuh"
#include "../../include/lutamm.h"
#include <cuda_fp16.h>

namespace lutamm {

namespace {

constexpr int kThreads = 128;
constexpr uint32_t kTmemColumns = 128;
constexpr uint32_t kBlind = 7;   // tiles scanned without a look at the scores before one that is looked at
constexpr float kUnit = 5.9604644775390625e-08f;   // 2^-24

template <int V, int CT, int CC>
struct Form {
    static constexpr int kUnits = (3 * V + 2 + 15) / 16 * 2;                      // 16-byte units of a codebook's axis
    static constexpr int kVec = CC * V / 4;                                       // float4 of a token; items of a thread
    static constexpr int kSpan = V / 4;                                           // ... of a codebook
    static constexpr int kWindow = CC * CT < 128 ? CC * CT : 128;                 // columns computed at once
    static constexpr int kRead = 64, kParts = kWindow / kRead, kCbPart = CT < kRead ? kRead / CT : 1;   // ... and read at once
    static constexpr int kWindows = CC * CT / kWindow, kCbWindow = kWindow / CT;
    static constexpr int kALead = kThreads * 16 + 16, kBLead = CC * CT * 16;      // bytes from unit to unit
    static constexpr int kABytes = CC * kUnits * kALead, kBBytes = kUnits * kBLead;
    static constexpr int kNormPitch = kThreads + 8;
    static constexpr int kWords = (CT + 31) / 32;                                 // of a mask of candidates
    static constexpr int kQueue = 32 * CC + 32;                                   // undecided (token, codebook) pairs of a warp: a tile's and fewer than 32 of earlier ones
    static constexpr int kTile = kVec * kNormPitch;                               // norms of a tile
    static constexpr size_t kSmem = 2 * kABytes + kBBytes + (2 * kTile + 4 * kQueue) * sizeof(float);
    static_assert(V % 4 == 0 && kVec == 4 && CC <= 4 && CT >= 32 && CC * CT % kWindow == 0 && kWindow % CT == 0 && CT % 16 == 0 && kWindow % kRead == 0, "");
    static_assert(kBLead / 16 < 1 << 14, "");
};

__device__ __forceinline__ uint64_t plain_desc(uint32_t addr, uint32_t lead) {   // K-major, no swizzle: 8 rows x 16 bytes are contiguous
    uint64_t d = 0;
    d |= static_cast<uint64_t>((addr & 0x3FFFFu) >> 4);
    d |= static_cast<uint64_t>(lead >> 4) << 16;      // to the next 16 bytes of the contraction axis
    d |= static_cast<uint64_t>(128u >> 4) << 32;      // to the next eight rows
    d |= static_cast<uint64_t>(1) << 46;
    return d;
}
// kind::f16 with f16 operands and fp32 sums, both K-major
__host__ __device__ constexpr uint32_t f16_idesc(uint32_t n) { return (1u << 4) | ((n >> 3) << 17) | ((kThreads >> 4) << 24); }

__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ uint32_t bits(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ void split(float2 a, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __float22half2_rn(a);
    const float2 back = __half22float2(h);
    hi = bits(h);
    lo = bits(__float22half2_rn(__fadd2_rn(a, make_float2(-back.x, -back.y))));
}
__device__ __forceinline__ uint32_t split_half(float a) {   // hi in the low half, lo in the high one
    const __half h = __float2half_rn(a);
    return bits(__halves2half2(h, __float2half_rn(a - __half2float(h))));
}
constexpr uint32_t kOnes = 0x3C003C00u;

// One bit per key that lies below the threshold, like below(): the upper half of the keys by saturating multiply-adds, 1
// or 0 each, that a second one weighs and sums in the mantissa of 2^23, so that they share the ALU's work with the FMA
// pipe.  (2^100 (thr - key) is 0 or beyond 1: both are multiples of 2^-60, and below 2^26.)
__device__ __forceinline__ uint32_t below_both(const float (&k)[32], float thr) {
    float lo[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) lo[i] = k[i];
    const float big = __int_as_float((127 + 100) << 23), far = thr * big;
    float sum = 8388608.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        float t;
        asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(t) : "f"(k[16 + i]), "f"(-big), "f"(far));
        sum = fmaf(t, (float)(1 << i), sum);
    }
    return __byte_perm(below<16>(lo, thr), __float_as_uint(sum), 0x5410);
}

// The reference's scan (ccs_scan.cuh) with the centroids straight from global memory (L1), 32 numbers in flight, two
// components per packed instruction.  c - x for x - c: the squares are the same.
template <int V, int CT>
__device__ __forceinline__ uint32_t scan(const float* __restrict__ xp, const float* __restrict__ cp) {
    float x[V];   // negated
#pragma unroll
    for (int d = 0; d < V; d += 4) {
        const float4 q = __ldg(reinterpret_cast<const float4*>(xp + d));
        x[d] = -q.x; x[d + 1] = -q.y; x[d + 2] = -q.z; x[d + 3] = -q.w;
    }
    float mn = 0.f;
    uint32_t best = 0;
    constexpr int kGroup = 32 / V;
    static_assert(CT % kGroup == 0 && 32 % V == 0, "");
#pragma unroll 1
    for (uint32_t g = 0; g < CT; g += kGroup) {
        float k[32];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float4 q = __ldg(reinterpret_cast<const float4*>(cp + g * V) + i);
            k[4 * i] = q.x; k[4 * i + 1] = q.y; k[4 * i + 2] = q.z; k[4 * i + 3] = q.w;
        }
#pragma unroll
        for (int c = 0; c < kGroup; ++c) {
            float acc = 0.f;
#pragma unroll
            for (int d = 0; d < V; d += 2) {
                const float2 e = __fadd2_rn(make_float2(k[c * V + d], k[c * V + d + 1]), make_float2(x[d], x[d + 1]));
                const float2 sq = __fmul2_rn(e, e);
                acc = d == 0 ? sq.x : __fadd_rn(acc, sq.x);   // 0 + sq.x is exact
                acc = __fadd_rn(acc, sq.y);
            }
            const bool take = (c == 0 && g == 0) || __fsub_rn(mn, acc) > kEps;   // false for NaN: keeps the earlier index
            mn = take ? acc : mn;
            best = take ? g + c : best;
        }
    }
    return best;
}

template <int V, int CT, int CC>
__global__ void __launch_bounds__(kThreads, 4)
ccs_umma_kernel(const float* __restrict__ x, const float* __restrict__ cent, uint8_t* __restrict__ out, uint32_t M, uint32_t K,
                uint32_t CB, uint32_t tiles, uint32_t tiles_per_cta, uint32_t* dev_err) {
    using F = Form<V, CT, CC>;
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char* s_a = smem;                                                   // [2]
    unsigned char* s_b = smem + 2 * F::kABytes;
    float* s_norm = reinterpret_cast<float*>(s_b + F::kBBytes);                  // [2][kVec][kNormPitch]
    __shared__ uint32_t s_top[CC];          // max |c|^2, scaled, as bits (NaN and infinity sort last)
    __shared__ float s_margin[8];           // of the centroids and of what does not depend on the magnitude
    __shared__ uint32_t s_unsound;          // codebooks whose centroids are not finite, or too far apart for f16
    __shared__ uint32_t s_largest;          // largest finite |component| as bits
    __shared__ uint32_t s_tmem, s_abort, s_read;
    __shared__ __align__(8) uint64_t s_bar;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    uint32_t* queue = reinterpret_cast<uint32_t*>(s_norm + 2 * F::kTile) + warp * F::kQueue;
    const uint32_t cb0 = blockIdx.x * CC;
    const uint32_t t0 = blockIdx.y * tiles_per_cta, t1 = min(tiles, t0 + tiles_per_cta);

    if (warp == 0) {
        tmem_alloc(smem_u32(&s_tmem), kTmemColumns);
        tmem_relinquish();
    }
    if (tid == 32) {
        mbar_init(smem_u32(&s_bar), 1);
        fence_barrier_init();
        s_abort = 0;
        s_largest = 0;
        s_unsound = 0;
        s_read = 0;
    }
    if (tid < CC) s_top[tid] = 0;
    __syncthreads();

    // The centroids, scaled and negated.
    const float* gc = cent + (size_t)cb0 * CT * V;
    {
        float top = 0.f;
        for (uint32_t e = tid; e < CC * CT * V; e += kThreads) {
            const float a = fabsf(__ldg(gc + e));
            if (a < __int_as_float(0x7f800000)) top = fmaxf(top, a);
        }
        atomicMax(&s_largest, __float_as_uint(top));
    }
    __syncthreads();
    float scale = 1.f;
    if (s_largest) {
        const int e = min(40, max(-40, 3 - ((int)(s_largest >> 23) - 127)));
        scale = __int_as_float((127 + e) << 23);
    }
    for (uint32_t r = tid; r < CC * CT; r += kThreads) {
        const uint32_t cb = r / CT;
        unsigned char* row = s_b + r * 16;
        uint32_t w[F::kUnits * 4];
#pragma unroll
        for (int i = 0; i < F::kUnits * 4; ++i) w[i] = 0;
        float cc = 0.f;
#pragma unroll
        for (int d = 0; d < V; d += 2) {
            const float2 c = make_float2(-scale * __ldg(gc + r * V + d), -scale * __ldg(gc + r * V + d + 1));
            cc = fmaf(c.x, c.x, cc);
            cc = fmaf(c.y, c.y, cc);
            uint32_t hi, lo;
            split(c, hi, lo);
            w[d / 2] = hi;
            w[V / 2 + d / 2] = lo;
            w[V + d / 2] = hi;
        }
        w[3 * V / 2] = split_half(0.5f * cc);
#pragma unroll
        for (int u = 0; u < F::kUnits; ++u)
            *reinterpret_cast<uint4*>(row + u * F::kBLead) = make_uint4(w[4 * u], w[4 * u + 1], w[4 * u + 2], w[4 * u + 3]);
        atomicMax(&s_top[cb], __float_as_uint(cc));
    }
    if constexpr (V > 4) {   // what no activation overwrites: the ones behind the components, and zeros
        for (uint32_t i = tid; i < 2 * CC * kThreads; i += kThreads) {
            unsigned char* p = s_a + (i / kThreads) * F::kUnits * F::kALead + (i % kThreads) * 16;
#pragma unroll
            for (int k = 3 * V / 2; k < F::kUnits * 4; ++k)
                *reinterpret_cast<uint32_t*>(p + (k / 4) * F::kALead + (k % 4) * 4) = k == 3 * V / 2 ? kOnes : 0u;
        }
    }
    __syncthreads();
    constexpr float kFactor = (24 * V + 64) * kUnit;
    if (tid < CC) {
        const float top = __uint_as_float(s_top[tid]);
        if (!(top < 1e6f)) atomicOr(&s_unsound, 1u << tid);
        s_margin[tid] = fmaf(kFactor, top, fmaf(kMarginBase * scale, scale, 1.2e-6f * V));
    }
    // Only now may the kernel behind come early: all CTAs hold their columns of tensor memory, which that kernel wants all of.
    pdl_launch_dependents();
    pdl_wait_prior_grid();

    const uint32_t tmem = s_tmem, bar = smem_u32(&s_bar);
    const uint32_t a_addr = smem_u32(s_a), b_addr = smem_u32(s_b);
    volatile uint32_t* abort_word = &s_abort;

    // A warp's items are those of its own 32 tokens, so that the norms stay within the warp.
    float4 nx[F::kVec];
    auto fetch = [&](uint32_t tile) {   // rows past the end repeat the last one (their results are not stored)
#pragma unroll
        for (int i = 0; i < F::kVec; ++i) {
            const uint32_t item = i * 32 + lane, row = warp * 32 + item / F::kVec, col = item % F::kVec;
            nx[i] = __ldg(reinterpret_cast<const float4*>(x + (size_t)min(tile * kThreads + row, M - 1) * K + cb0 * V) + col);
        }
    };
    auto convert = [&](uint32_t side) {
        float* norm = s_norm + side * F::kTile;
        unsigned char* a = s_a + side * F::kABytes;
#pragma unroll
        for (int i = 0; i < F::kVec; ++i) {
            const uint32_t item = i * 32 + lane, row = warp * 32 + item / F::kVec, col = item % F::kVec;
            const float2 s = make_float2(scale, scale);
            const float2 p = __fmul2_rn(make_float2(nx[i].x, nx[i].y), s), q = __fmul2_rn(make_float2(nx[i].z, nx[i].w), s);
            const float2 sq = __ffma2_rn(q, q, __fmul2_rn(p, p));
            norm[col * F::kNormPitch + row] = sq.x + sq.y;
            uint32_t ph, pl, qh, ql;
            split(p, ph, pl);
            split(q, qh, ql);
            unsigned char* dst = a + row * 16;
            if constexpr (V == 4) {
                *reinterpret_cast<uint4*>(dst + 2 * col * F::kALead) = make_uint4(ph, qh, ph, qh);
                *reinterpret_cast<uint4*>(dst + (2 * col + 1) * F::kALead) = make_uint4(pl, ql, kOnes, 0);
            } else {
                const uint32_t cb = col / (V / 4), j = col % (V / 4);
                auto at = [&](uint32_t k) { return dst + (cb * F::kUnits + k / 4) * F::kALead + (k % 4) * 4; };   // k: 32-bit word of the axis
                *reinterpret_cast<uint2*>(at(2 * j)) = make_uint2(ph, qh);
                *reinterpret_cast<uint2*>(at(V / 2 + 2 * j)) = make_uint2(ph, qh);
                *reinterpret_cast<uint2*>(at(V + 2 * j)) = make_uint2(pl, ql);
            }
        }
        fence_proxy_async_smem();
    };
    auto issue = [&](uint32_t side, uint32_t w) {   // scores of window w; one warp, converged
        tc_fence_after_sync();
        if (elect_one()) {
#pragma unroll
            for (int g = 0; g < F::kWindow / CT; ++g) {
                const uint32_t n = w * (F::kWindow / CT) + g;
                const uint64_t a = plain_desc(a_addr + side * F::kABytes + n * F::kUnits * F::kALead, F::kALead);
                const uint64_t b = plain_desc(b_addr + n * CT * 16, F::kBLead);
#pragma unroll
                for (int k = 0; k < F::kUnits / 2; ++k)
                    umma_f16(tmem + g * CT, a + k * (2 * F::kALead >> 4), b + k * (2 * F::kBLead >> 4), f16_idesc(CT), k > 0);
            }
            umma_commit(bar);
        }
        __syncwarp();
    };
    // This warp has read a window; the last of the four has the next one computed.  All of them converted the next
    // tile before they read any window of this one.
    auto release = [&](uint32_t side, uint32_t w, bool more) {
        tc_fence_before_sync();
        __syncwarp();
        uint32_t n = 0;
        if (lane == 0)
            asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;" : "=r"(n) : "r"(smem_u32(&s_read)) : "memory");
        n = __shfl_sync(0xFFFFFFFFu, n, 0);
        __syncwarp();
        if ((n & 3u) == 3u && (w + 1 < F::kWindows || more)) issue(w + 1 < F::kWindows ? side : side ^ 1u, (w + 1) % F::kWindows);
    };
    uint32_t queued = 0;
    // Settles the queue, 32 pairs at a time, until fewer than `least` are left.
    auto settle_all = [&](uint32_t least) {
        __syncwarp();
        uint32_t done = 0;
#pragma unroll 1
        for (; done + least <= queued; done += 32) {
            if (done + lane < queued) {
                const uint32_t q = queue[done + lane], m = t0 * kThreads + q / 8, b = q % 8;
                out[(size_t)m * CB + cb0 + b] = (uint8_t)scan<V, CT>(x + (size_t)m * K + (cb0 + b) * V, gc + b * (CT * V));
            }
        }
        const uint32_t rest = queued > done ? queued - done : 0;
        const uint32_t keep = lane < rest ? queue[done + lane] : 0;
        __syncwarp();
        if (lane < rest) queue[lane] = keep;
        queued = rest;
        __syncwarp();
    };

    bool ok = true;
    uint32_t phase = 0;
    if (t0 < t1) {
        fetch(t0);
        convert(0);
    }
    __syncthreads();
    if (t0 < t1 && warp == 0) issue(0, 0);
    if (t0 + 1 < t1) fetch(t0 + 1);
    uint32_t blind = 0;   // tiles to come for which the scores are not looked at
    for (uint32_t tile = t0; tile < t1; ++tile) {
        const uint32_t side = (tile - t0) & 1u;
        const bool more = tile + 1 < t1;
        const float* norm = s_norm + side * F::kTile;
        if (more) {
            convert(side ^ 1u);
            if (tile + 2 < t1) fetch(tile + 2);
        }
        __syncwarp();
        const uint32_t m = tile * kThreads + tid;
        float all = 0.f;
#pragma unroll
        for (int i = 0; i < F::kVec; ++i) all += norm[i * F::kNormPitch + tid];
        const uint32_t unsound = m >= M ? 0u : all < (float)(1 << 29) ? s_unsound : 0xFFu;
        uint32_t word = 0;
        auto margin = [&](uint32_t b) {
            float xx = 0.f;
#pragma unroll
            for (int i = 0; i < F::kSpan; ++i)
                xx += norm[(b * F::kSpan + i) * F::kNormPitch + tid];
            return fmaf(kFactor, xx, s_margin[b]);
        };
        auto defer = [&](uint32_t b, bool undecided) {   // all lanes
            const uint32_t who = __ballot_sync(0xFFFFFFFFu, undecided && m < M);
            if (undecided && m < M) queue[queued + __popc(who & ((1u << lane) - 1))] = ((tile - t0) * kThreads + tid) * 8 + b;
            queued += __popc(who);
        };
        const uint32_t before = queued;
        if (blind) {   // most pairs of an earlier tile were undecided: its scan at once
            --blind;
#pragma unroll 1
            for (uint32_t w = 0; w < F::kWindows && ok; ++w) {
                ok = mbar_wait_warp(bar, phase, abort_word);
                if (!ok) break;
                phase ^= 1u;
                release(side, w, more);
            }
#pragma unroll 1
            for (uint32_t b = 0; b < (m < M && ok ? CC : 0); ++b)
                word |= scan<V, CT>(x + (size_t)m * K + (cb0 + b) * V, gc + b * (CT * V)) << (8 * b);
        } else
#pragma unroll 1
        for (uint32_t w = 0; w < F::kWindows; ++w) {
            ok = mbar_wait_warp(bar, phase, abort_word);
            if (!ok) break;   // a warp that leaves issues nothing more, and the others' waits see the abort word
            phase ^= 1u;
            tc_fence_after_sync();
            float least[F::kParts];
            uint32_t cand[F::kCbWindow][F::kWords], several = (unsound >> (w * F::kCbWindow)) & ((1u << F::kCbWindow) - 1);
            uint32_t got = 0;
#pragma unroll
            for (int part = 0; part < F::kParts; ++part) {
                uint32_t raw[2][32];
                const uint32_t from = tmem + ((warp * 32) << 16) + part * F::kRead;
                tmem_ld_32x32b_x32(from, raw[0]);
                tmem_ld_32x32b_x32(from + 32, raw[1]);
                tmem_ld_wait();
                if (part == F::kParts - 1) release(side, w, more);
                constexpr int kG = CT < 64 ? CT : 64;
#pragma unroll
                for (int i = 0; i < F::kCbPart; ++i) {
                    const int j = CT <= 64 ? part * F::kCbPart + i : 0;
                    float k[kG];
#pragma unroll
                    for (int c = 0; c < kG; ++c) k[c] = __uint_as_float(raw[(i * CT + c) / 32][(i * CT + c) % 32]);
                    least[part] = min_of(k);
                    const float thr = least[part] + margin(w * F::kCbWindow + j);
                    if constexpr (CT == 32) {
                        cand[j][0] = below_both(k, thr);
                        several |= all_but_lowest(cand[j][0]);
                        got |= (high_bit(cand[j][0]) & 31u) << (8 * j);
                    } else {
                        constexpr int kAt = CT == 64 ? 0 : 2;
                        float lo[32], hi[32];
#pragma unroll
                        for (int c = 0; c < 32; ++c) { lo[c] = k[c]; hi[c] = k[32 + c]; }
                        cand[j][kAt * part] = below_both(lo, thr);
                        cand[j][kAt * part + 1] = below_both(hi, thr);
                        if constexpr (CT == 64) {
                            const uint32_t l = cand[j][0], h = cand[j][1];
                            several |= all_but_lowest(l) | all_but_lowest(h) | (l ? h : 0u);
                            got |= (high_bit(l ? l : h) & 31u | (l ? 0u : 32u)) << (8 * j);
                        }
                    }
                }
            }
            if constexpr (CT == 128) {   // a half's candidates stay if its smallest score is within the margin of the other's
                const float bound = fminf(least[0], least[1]) + margin(w);
                uint32_t found = 0, base = 0;
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    cand[0][g] = least[g / 2] < bound ? cand[0][g] : 0u;
                    several |= all_but_lowest(cand[0][g]) | (cand[0][g] ? found : 0u);
                    base = cand[0][g] ? 32 * g : base;
                    found = cand[0][g] ? cand[0][g] : found;
                }
                got = base + (high_bit(found) & 31u);
            }
            word |= F::kWindows == 1 ? got : got << (8 * F::kCbWindow * w);
            if (__any_sync(0xFFFFFFFFu, several != 0)) {
#pragma unroll 1
                for (int j = 0; j < F::kCbWindow; ++j) {
                    uint32_t c[F::kWords], rest = 0, seen = 0;
#pragma unroll
                    for (int g = 0; g < F::kWords; ++g) {
#pragma unroll
                        for (int i = 0; i < F::kCbWindow; ++i) c[g] = i == 0 || i == j ? cand[i][g] : c[g];
                        rest |= all_but_lowest(c[g]) | (c[g] ? seen : 0u);
                        seen |= c[g];
                    }
                    defer(w * F::kCbWindow + j, ((unsound >> (w * F::kCbWindow + j)) & 1u) || rest != 0);
                }
            }
        }
        if (!ok) break;
        if (m < M) {
            uint8_t* o = out + (size_t)m * CB + cb0;
            if constexpr (CC == 4) *reinterpret_cast<uint32_t*>(o) = word;
            else *reinterpret_cast<uint16_t*>(o) = (uint16_t)word;
        }
        if (queued - before > 24 * CC) blind = kBlind;   // three quarters: from there on the scores cost more than they save
        if (queued >= 32) settle_all(32);
    }
    if (queued && ok) settle_all(1);
    tc_fence_before_sync();
    __syncthreads();
    if (s_abort) {
        if (tid == 0) {   // instructions that may still be in flight have a bounded time to end before their memory is handed back
            const long long start = clock64();
            while (clock64() - start < 200000) {}
            report_error(dev_err, 5u);
        }
        __syncthreads();
    }
    if (warp == 0) {
        tc_fence_after_sync();
        tmem_dealloc(tmem, kTmemColumns);
    }
}

uint32_t sm_count() {
    static const uint32_t n = [] {
        int dev = 0, v = 0;
        cudaGetDevice(&dev);
        return cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && v > 0 ? (uint32_t)v : 148u;
    }();
    return n;
}

// Tiles of a CTA: runs of equal length in up to four waves, one more tile standing for what a CTA spends on its centroids.
// `used`: the part of that time that the GPU's CTAs spend on tokens.
template <int V, int CT, int CC>
uint32_t plan_run(const CcsArgs& a, float* used) {
    constexpr uint32_t kFit = (uint32_t)(227 * 1024 / (Form<V, CT, CC>::kSmem + 1024 + 256)), kPerSm = kFit < 4 ? kFit : 4;   // (1 KB a CTA is the system's)
    const uint32_t groups = a.CB / CC, tiles = (a.M + kThreads - 1) / kThreads;
    const uint64_t resident = (uint64_t)kPerSm * sm_count();
    uint32_t run = tiles;
    uint64_t least = ~0ull;
    for (uint64_t waves = 1; waves <= 4; ++waves) {
        const uint64_t want = waves * resident / groups, y = want < 1 ? 1 : want > tiles ? tiles : want;
        const uint32_t r = (uint32_t)((tiles + y - 1) / y);
        const uint64_t ctas = (uint64_t)groups * ((tiles + r - 1) / r), cost = (ctas + resident - 1) / resident * (r + 1);
        if (cost < least) { least = cost; run = r; }
    }
    *used = (float)groups * (float)a.M / (float)kThreads / ((float)resident * (float)least);
    return run;
}

template <int V, int CT, int CC>
cudaError_t run(const CcsArgs& a, cudaStream_t s) {
    using F = Form<V, CT, CC>;
    auto k = ccs_umma_kernel<V, CT, CC>;
    static SmemOptIn memo;
    cudaError_t e = allow_smem(memo, k, (int)F::kSmem);
    if (e != cudaSuccess) return e;
    float used;
    const uint32_t run = plan_run<V, CT, CC>(a, &used), groups = a.CB / CC, tiles = (a.M + kThreads - 1) / kThreads;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(groups, (tiles + run - 1) / run);
    if (cfg.gridDim.y > 65535u) return cudaErrorInvalidValue;
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = F::kSmem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, a.x, a.centroid, static_cast<uint8_t*>(a.idx_out), a.M, a.K, a.CB, tiles, run, a.dev_err);
}

// (sub-vector length, centroids, codebooks of a CTA)
#define LUTAMM_CCS_UMMA_INSTANCES(X) X(4, 32, 4) X(4, 64, 4) X(4, 128, 4) X(8, 32, 2) X(8, 64, 2)
// In calls of few scores the prologue (tensor memory, the centroids) costs as much as it saves, and so do the empty waves
// of few tokens of very many codebooks.  Times of ccs_tile_kernel over those of this one, with a 192-column contraction, over
// 48 to 1536 codebooks:
//     scores             100 M           50 M            25 M            12 M
//     32 centroids       1.01 to 1.23    1.00 to 1.21    0.97 to 1.10    0.92 to 1.06
//     64 and 128         1.15 to 1.54    1.09 to 1.42    1.06 to 1.37    1.04 to 1.50
//     128, v = 4, 390 x 2560, 0.37 of the time used 1.14; 768 x 2560, 0.54 1.07; 512 x 2048, 0.69 1.30; 1400 x 2048, 0.79 1.32
// Both lines were drawn for this kernel when it settled undecided pairs centroid by centroid (0.95 at 50 M, 0.86 and 0.93 in
// the first two of the last row); for 64 centroids and more they now lie higher than they need.
constexpr float kLeastUsed = 0.6f;
constexpr uint64_t kFewestScores = 96000000;

}  // namespace

bool ccs_umma_takes(const CcsArgs& a) {
    if (!a.dev_err || a.format != LUTAMM_INDEX_U8_ROWMAJOR || a.tokens_per_thread) return false;
    if ((uint64_t)a.M * a.CB * a.CT < kFewestScores || reinterpret_cast<uintptr_t>(a.x) % 16 || reinterpret_cast<uintptr_t>(a.centroid) % 16 || a.K % 4) return false;
#define LUTAMM_CCS_UMMA(V_, CT_, CC_) \
    if (a.v == V_ && a.CT == CT_) {                                                                                     \
        float used = 0.f;                                                                                               \
        if (a.CB % CC_ == 0 && reinterpret_cast<uintptr_t>(a.idx_out) % CC_ == 0) plan_run<V_, CT_, CC_>(a, &used);      \
        return used >= kLeastUsed;                                                                                      \
    }
    LUTAMM_CCS_UMMA_INSTANCES(LUTAMM_CCS_UMMA)
#undef LUTAMM_CCS_UMMA
    return false;
}

cudaError_t launch_ccs_umma(const CcsArgs& a, cudaStream_t s) {
#define LUTAMM_CCS_UMMA(V_, CT_, CC_) \
    if (a.v == V_ && a.CT == CT_) return run<V_, CT_, CC_>(a, s);
    LUTAMM_CCS_UMMA_INSTANCES(LUTAMM_CCS_UMMA)
#undef LUTAMM_CCS_UMMA
    return cudaErrorInvalidValue;
}

}  // namespace lutamm
