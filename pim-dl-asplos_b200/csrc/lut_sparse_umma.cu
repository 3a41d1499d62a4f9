// Steps 2+3 of the AMM on CTA pairs with the one-hot operand in the tensor cores' 2:4 sparse form.
//
// The same contraction as lut_onehot_umma.cu - acc[M x N] = OneHot[M x (CB*CT)] * LUT[(CB*CT) x N], exact in int32 -
// at twice its rate.  A one-hot row has at most one non-zero per codebook, so it is 2:4 sparse: of every four positions
// the operand stores two bytes and a nibble of metadata that says which two positions they stand for (build_row).
//
// Why pairs.  The sparse instruction eats 256 bytes of the contraction axis a row in the time the dense one eats
// 128, and a LUT byte is read from L2 and from shared memory once per row tile: with 128 rows a tile shared memory
// would have to deliver 128 B/clk to the tensor core alone, beside the 128 B/clk that the copies fill.  A pair of
// CTAs (cta_group::2) works on 256 rows and each SM loads and reads half of the LUT slab: 64 + 64 B/clk.
//
// Otherwise the structure of the dense kernel: persistent, one pair per two SMs walking 256-token x N_TILE items,
// accumulators double-buffered in tensor memory, every slot of both rings with one producer and one consumer.  Per CTA:
//   warps 0-1     copy the CTA's half of a LUT slab (N_TILE/2 rows x 256 bytes); bytes count on the leader's barrier
//   warp 2        copies the index bytes of the CTA's rows, a few slabs at a time
//   warps 3-6     leader only: four tcgen05.mma.sp per slab, slab x by warp 3 + x % 4, in turn (below)
//   warps 7-22    four groups of four warps: the operand of the CTA's 128 rows, straight from the uint8 indices;
//                 group k takes every fourth slab, one row per thread, in registers: a table in shared memory would
//                 compete with the slabs for its bandwidth
//   warps 23-26   epilogue: tcgen05.ld, dequantise, swizzled staging, tiled bulk stores; clears the accumulator
//
// What bounds it.  With a long codebook axis (16384 x 2048 codebooks of 16 -> 4096) a slab takes 220 ns, 340-380 cycles
// at the 1.55-1.7 GHz that the power cap leaves, against 320 of the tensor pipe: 1254 -> 648 us, 6.8 P operations/s of the
// dense contraction (4.57 is the dense pipe's peak).  With a short one (BERT-base QKV, 24 slabs a tile, 12608 tokens:
// 118 -> 65 us) it is the epilogue of the tile before, 0.93 us per 32 columns, beside the main loop.  Steps on the way, at
// 12608 x 384 -> 3072 (dense 160 us): arrivals with .release.cluster, which waits for the builder's loads, 160; default
// scope 108; two copying threads 105; an issuing warp per operand slot 99; index tiles through the copy engine 84.
#include "kernels.h"
#include "ptx.cuh"
#include "epilogue.cuh"

namespace lutamm {

namespace {

constexpr uint32_t kRows = 128;                // rows of a CTA: half a tile
constexpr uint32_t kSlab = 256;                // positions of the contraction axis per ring slot
constexpr uint32_t kGroups = 4, kCopyWarps = 2, kIndexWarps = 1, kMmaWarps = 4, kEpiWarps = 4;
constexpr uint32_t kFirstMma = kCopyWarps + kIndexWarps, kFirstBuilder = kFirstMma + kMmaWarps, kFirstEpi = kFirstBuilder + 4 * kGroups;
constexpr uint32_t kThreads = (kFirstEpi + kEpiWarps) * 32;   // 864
// Wider tiles than 160 columns are for launches of one tile per pair: a second accumulator would leave no room for slots.
__host__ __device__ constexpr uint32_t accumulators(uint32_t n_tile) { return n_tile > 160 ? 1 : 2; }
// operand slots, 32 columns of bytes and 2 of metadata each: what the accumulators leave, in multiples of the groups
__host__ __device__ constexpr uint32_t operand_slots(uint32_t n_tile) { return (512 - accumulators(n_tile) * n_tile) / 34 >= 8 ? 8 : 4; }
constexpr uint32_t kMaxASlots = 8;
constexpr uint32_t kMaxBSlots = 16;
constexpr uint32_t kStageBytes = 32 * 128;     // a 32 x 32 fp32 block
constexpr uint32_t kStages = 2;                // per epilogue warp
constexpr uint32_t kIdxStages = 3;
__host__ __device__ constexpr uint32_t stage_blocks(uint32_t n_tile) { return accumulators(n_tile) == 1 ? 0 : kEpiWarps * kStages; }
constexpr uint32_t kNumBarriers = 2 * kMaxASlots + 2 * kMaxBSlots + 4 + 2 * kIdxStages + 4 + kMmaWarps;

// A stage of index bytes: 128 rows of `idx_width` bytes, for `idx_slabs` slabs.
__host__ __device__ constexpr uint32_t idx_width(int lg) { return lg == 3 ? 64u : lg <= 6 ? 4u * (256u >> lg) : 16u; }
__host__ __device__ constexpr uint32_t idx_slabs(int lg) { return (idx_width(lg) << lg) / kSlab; }

struct SparseParams {
    LutArgs a;
    uint32_t slabs;          // of the whole codebook axis
    uint32_t split, per;     // slices of it, slabs of a slice
    uint32_t b_slots, tiles_m, tiles_n, group_m, one_tile, early_trigger, fresh_table;
    uint4* partial;          // split > 1: [tile][CTA][quadrant][slice][chunk of 32 columns][4 columns][row] int32
    uint32_t* counters;      // split > 1: [tile][CTA][quadrant] x (slices arrived, slices done), zero between launches
    uint32_t* dev_err;
};

// Out = one word per combination of the index bits in BITS (highest first): in & (bit or its complement), two bits per
// three-input operation.  A word holds bytes of several codebooks; `in` carries at most bit 0 of each, so what else the
// shifted indices hold does not matter.
template <int N>
__device__ __forceinline__ void split1(const uint32_t (&in)[N], uint32_t b, uint32_t (&out)[2 * N]) {
#pragma unroll
    for (int i = 0; i < N; ++i) { out[2 * i] = in[i] & ~b; out[2 * i + 1] = in[i] & b; }
}
template <int N>
__device__ __forceinline__ void split2(const uint32_t (&in)[N], uint32_t b1, uint32_t b0, uint32_t (&out)[4 * N]) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
        out[4 * i] = in[i] & ~b1 & ~b0; out[4 * i + 1] = in[i] & ~b1 & b0;
        out[4 * i + 2] = in[i] & b1 & ~b0; out[4 * i + 3] = in[i] & b1 & b0;
    }
}

// The operand of one row's slab from its 256 / CT index bytes: 128 stored bytes (w) and the metadata of 64 positions of
// the axis (m), which repeats for all four instructions of the slab.
//
// Stored byte p = d * codebooks + codebook, d being the centroid index without its bit H: bytes of four codebooks share
// a word, so a word is the AND of a few (complemented) bits of four packed indices - one three-input operation - where
// codebook-major bytes would take two shifts and an extraction per codebook.  Positions 2p and 2p + 1 of the axis belong
// to byte p: the index's bit H chooses, through the metadata nibble of the pair of bytes (2g, 2g + 1): the first stands
// for position 0 or 1 of four, the second for 2 or 3.  The table is laid out to match (launch_sparse_table, H = 1), or its
// rows are copied in that order (the highest bit: then the rest of the index counts rows, and four dimensions say it all).
//
// An index that is out of range (they may come from a caller) stores nothing.
template <int LG, int H>
__device__ __forceinline__ void build_row(const uint32_t (&raw)[LG == 3 ? 8 : 4], uint32_t (&w)[32], uint32_t (&m)[2]) {
    constexpr int kCbs = 256 >> LG, kQ = kCbs >= 4 ? kCbs / 4 : 1;   // codebooks, words of packed indices
    constexpr uint32_t kOnes = 0x01010101u, kBeyond = LG == 8 ? 0u : ((0xFFu << LG) & 0xFFu) * kOnes;
    uint32_t v[kQ], valid[kQ], top[kQ], any = 0;
#pragma unroll
    for (int q = 0; q < kQ; ++q) {
        if constexpr (LG == 8) v[q] = (raw[0] & 0xFFu) * kOnes;
        else if constexpr (LG == 7) v[q] = __byte_perm(raw[0], 0, 0x1010);
        else v[q] = raw[q];
        any |= v[q] & kBeyond;
        valid[q] = kOnes;
        // bits 0, 2, 4, 6 of the top byte: bit H of the four indices
        top[q] = ((v[q] >> H) & kOnes) * 0x01041040u;
    }
    if (LG < 8 && any) {
        constexpr uint32_t kRange = 1u << (8 - LG);
#pragma unroll
        for (int q = 0; q < kQ; ++q) valid[q] = ((kRange * kOnes - ((v[q] & kBeyond) >> LG)) >> (8 - LG)) & kOnes;
    }
#pragma unroll
    for (int q = 0; q < kQ; ++q) {
        const uint32_t x = v[q];
        auto bit = [x](int i) { return x >> (i >= H ? i + 1 : i); };   // bit i of d at bit 0 of the bytes
        if constexpr (LG == 3) {
            uint32_t in[1] = {valid[q]}, o[4];
            split2(in, bit(1), bit(0), o);
#pragma unroll
            for (int d = 0; d < 4; ++d) w[d * kQ + q] = o[d];
        } else if constexpr (LG == 4) {
            uint32_t in[1] = {valid[q]}, t[2], o[8];
            split1(in, bit(2), t);
            split2(t, bit(1), bit(0), o);
#pragma unroll
            for (int d = 0; d < 8; ++d) w[d * kQ + q] = o[d];
        } else if constexpr (LG == 5) {
            uint32_t in[1] = {valid[q]}, t[4], o[16];
            split2(in, bit(3), bit(2), t);
            split2(t, bit(1), bit(0), o);
#pragma unroll
            for (int d = 0; d < 16; ++d) w[d * kQ + q] = o[d];
        } else {
            // 32 words of one index word: five bits; what is left of d lies within the word
            uint32_t in[1], t[2], u[8];
            if constexpr (LG == 6) in[0] = valid[q];
            else if constexpr (LG == 7) in[0] = valid[q] & ~(x ^ 0x01010000u);   // bytes: (d even) cb 0, 1, (d odd) cb 0, 1
            else in[0] = 1u << (8 * (((bit(1) & 1u) << 1) | (x & 1u)));
            split1(in, bit(LG - 2), t);
            split2(t, bit(LG - 3), bit(LG - 4), u);
            split2(u, bit(LG - 5), bit(LG - 6), w);
        }
    }
    uint32_t meta[2];
    if constexpr (LG == 3) {
        meta[0] = __byte_perm(__byte_perm(top[0], top[1], 0x0073), __byte_perm(top[2], top[3], 0x0073), 0x5410);
        meta[1] = __byte_perm(__byte_perm(top[4], top[5], 0x0073), __byte_perm(top[6], top[7], 0x0073), 0x5410);
    } else if constexpr (LG == 4) {
        meta[0] = meta[1] = __byte_perm(__byte_perm(top[0], top[1], 0x0073), __byte_perm(top[2], top[3], 0x0073), 0x5410);
    } else if constexpr (LG == 5) {
        meta[0] = meta[1] = __byte_perm(top[0], top[1], 0x7373);
    } else if constexpr (LG == 6) {
        meta[0] = meta[1] = __byte_perm(top[0], 0, 0x3333);
    } else {   // one nibble: (first codebook, second codebook), or the one codebook twice; the top byte holds it twice
        meta[0] = meta[1] = __byte_perm(top[0], 0, 0x3333);
    }
    m[0] = meta[0] | 0x88888888u;
    m[1] = meta[1] | 0x88888888u;
}

// One decision for all values: decided per value, the branches would part the code that has to overlap.
template <int N>
__device__ __forceinline__ void activate_all(float (&o)[N], uint32_t act) {
    if (act == 1u) {
#pragma unroll
        for (int q = 0; q < N; ++q) o[q] = activate_one(o[q], 1u);
    } else if (act) {
#pragma unroll
        for (int q = 0; q < N; ++q) o[q] = activate_one(o[q], 2u);
    }
}

// A work item: a tile, or a slice of its codebook axis.
struct SparseItem {
    uint32_t m0, n0, tile, z, begin, slabs;
};
template <bool SPLIT>
__device__ __forceinline__ SparseItem sparse_item(const SparseParams& p, uint32_t item, uint32_t n_tile, uint32_t rank) {
    const uint32_t tile = SPLIT ? item / p.split : item, z = SPLIT ? item % p.split : 0u, begin = SPLIT ? z * p.per : 0u;
    // row tiles in groups, column tiles within a group, row tiles of the group innermost
    const uint32_t g = tile / (p.group_m * p.tiles_n), in = tile - g * p.group_m * p.tiles_n, rows = min(p.group_m, p.tiles_m - g * p.group_m);
    const uint32_t tn = in / rows, tm = g * p.group_m + in - tn * rows;
    return {tm * (2 * kRows) + rank * kRows, tn * n_tile, tile, z, begin, SPLIT ? min(p.per, p.slabs - begin) : p.slabs};
}

// A slice's place in the partial sums of a quadrant (corner: tile, CTA, quadrant): per chunk of 32 columns 8 groups of four
// columns x 32 rows, coalesced both ways.
template <uint32_t N_TILE>
__device__ __forceinline__ uint4* partial_sums(const SparseParams& p, uint32_t corner, uint32_t z, uint32_t c, uint32_t lane) {
    return p.partial + (((size_t)corner * p.split + z) * (N_TILE / 32) + c) * 256 + lane;
}

// The end of a split tile.  Its slices are in progress together (the grid is one item per pair); for each quadrant of 32
// rows the epilogue warp of every slice waits, bounded, until all slices have stored, and then shares out the groups of
// four columns with the builder warps, who are done.  Eight loads in flight per warp: one slice or group after
// the other is a chain of L2 round trips (768 codebook slabs in three slices, 1024 tokens: 10 us of it with one warp).
// The last warp re-arms the counters.
constexpr uint32_t kSumWarps = 1 + kGroups;
template <uint32_t N_TILE>
__device__ __forceinline__ bool split_finish(const SparseParams& p, const SparseItem& it, uint32_t rank, uint32_t quad, uint32_t share, uint32_t lane,
                                             uint32_t sums_bar, volatile uint32_t* s_abort) {
    const LutArgs& a = p.a;
    const uint32_t corner = (it.tile * 2 + rank) * 4 + quad;
    uint32_t* ctr = p.counters + 2 * corner;   // [0] slices stored, [1] warps done
    bool go = true;
    if (share == 0) {
        if (lane == 0) {
            go = false;
            for (uint32_t spin = 0; spin < kWaitLimit && !go; ++spin) {
                go = *reinterpret_cast<volatile uint32_t*>(ctr) >= p.split;
                if ((spin & 63u) == 63u && *s_abort) break;
            }
            __threadfence();   // between the counter's value and the sums that it stands for, for everybody released here
            if (go) mbar_arrive(sums_bar + 8 * quad);
            else *s_abort = 1u;
        }
        go = __shfl_sync(0xffffffffu, go, 0);
        __syncwarp();   // ... in this warp too: a shuffle orders no memory
    } else {
        go = mbar_wait_warp<32>(sums_bar + 8 * quad, 0, s_abort);
    }
    if (!go) return false;
    const float lbcb = lut_bias_times_cb(a.lut_bias, a.CB);
    const uint32_t row = it.m0 + quad * 32 + lane;
    constexpr uint32_t kUnits = N_TILE / 4;   // groups of four columns
    const uint32_t step = p.split * kSumWarps;
    auto store = [&](uint32_t g, const uint4& sum) {
        const uint32_t n = it.n0 + 4 * g;
        if (n >= a.N || row >= a.M) return;   // N % 16 == 0: four columns are in or out together
        const float4 b4 = __ldg(reinterpret_cast<const float4*>(a.bias + n));
        float o[4] = {dequant_one((int32_t)sum.x, a.scale, lbcb, b4.x), dequant_one((int32_t)sum.y, a.scale, lbcb, b4.y),
                      dequant_one((int32_t)sum.z, a.scale, lbcb, b4.z), dequant_one((int32_t)sum.w, a.scale, lbcb, b4.w)};
        activate_all(o, a.act);
        *reinterpret_cast<float4*>(a.out + (size_t)row * a.N + n) = make_float4(o[0], o[1], o[2], o[3]);
    };
    auto load = [&](uint32_t g, uint32_t z) {
        return g < kUnits && z < p.split ? __ldcg(partial_sums<N_TILE>(p, corner, z, g >> 3, lane) + 32 * (g & 7u)) : make_uint4(0, 0, 0, 0);
    };
    auto add = [](uint4& s, const uint4& t) { s.x += t.x; s.y += t.y; s.z += t.z; s.w += t.w; };
    if (p.split <= 4) {   // two groups of up to four slices
        for (uint32_t g = it.z * kSumWarps + share; g < kUnits; g += 2 * step) {
            uint4 t0[4], t1[4];
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) { t0[k] = load(g, k); t1[k] = load(g + step, k); }
#pragma unroll
            for (uint32_t k = 1; k < 4; ++k) { add(t0[0], t0[k]); add(t1[0], t1[k]); }
            store(g, t0[0]);
            if (g + step < kUnits) store(g + step, t1[0]);
        }
    } else {
        for (uint32_t g = it.z * kSumWarps + share; g < kUnits; g += step) {
            uint4 sum = make_uint4(0, 0, 0, 0);
            for (uint32_t z0 = 0; z0 < p.split; z0 += 8) {   // integer sums: the order is immaterial
                uint4 t[8];
#pragma unroll
                for (uint32_t k = 0; k < 8; ++k) t[k] = load(g, z0 + k);
#pragma unroll
                for (uint32_t k = 0; k < 8; ++k) add(sum, t[k]);
            }
            store(g, sum);
        }
    }
    __syncwarp();
    if (lane == 0 && atomicAdd(ctr + 1, 1u) == p.split * kSumWarps - 1) { ctr[0] = 0u; ctr[1] = 0u; }
    return true;
}

// SPLIT: items are slices of a tile's codebook axis, one per pair.
// CANONICAL: the slabs come from the table as the caller has it, [codebook][centroid][N], columns contiguous: a slab is 256
// of its rows, in the order of the positions, by a four-dimensional copy (sparse_make_canonical_tmap), and the operand is
// column-major (MN-major) in shared memory.  For callers who have no room for the other layout, or use a table once: 512
// tokens, 384 codebooks of 16 -> 3072, the synchronous call 54 -> 25 us.  The copies move rows of 64 or 32 bytes where
// those of the other layout move 128, which costs nothing while the rows begin on sectors (a slab 0.16-0.2 us in a full
// round, like there); tiles are powers of two wide, as a row has to be one row of a swizzle pattern.
template <uint32_t N_TILE, int LG, bool SPLIT, bool CANONICAL>
__global__ void __launch_bounds__(kThreads, 1)
lut_sparse_kernel(const __grid_constant__ CUtensorMap lut_map, const __grid_constant__ CUtensorMap idx_map,
                  const __grid_constant__ CUtensorMap out_map, const SparseParams p) {
    constexpr uint32_t kHalfN = N_TILE / 2, kBBytes = kHalfN * kSlab;
    constexpr uint32_t kIdesc = umma_idesc_i8(2 * kRows, N_TILE, 1, 1) | kIdescSparse | (CANONICAL ? kIdescColumnMajorB : 0);
    static_assert(!CANONICAL || kHalfN == 32 || kHalfN == 64, "a row of a slab is one row of a swizzle pattern");
    constexpr uint32_t kASlots = operand_slots(N_TILE);
    constexpr bool kOne = accumulators(N_TILE) == 1;
    constexpr uint32_t kDataBase = accumulators(N_TILE) * N_TILE, kMetaBase = kDataBase + 32 * kASlots;   // tensor-memory columns
    static_assert(kMetaBase + 2 * kASlots <= 512, "tensor memory");

    constexpr uint32_t kIdxWidth = idx_width(LG), kIdxSlabs = idx_slabs(LG), kIdxBytes = kRows * kIdxWidth;

    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const uint32_t SB = p.b_slots;
    unsigned char* s_b = smem;                                        // [SB][2][kHalfN][128]
    unsigned char* s_stage = s_b + (size_t)SB * kBBytes;              // [4][kStages][32][128]
    unsigned char* s_idx = s_stage + stage_blocks(N_TILE) * kStageBytes;   // [kIdxStages][128][idx_width]
    float* s_bias = reinterpret_cast<float*>(s_idx + kIdxStages * kIdxBytes);   // [4][N_TILE]
    uint64_t* s_bar = reinterpret_cast<uint64_t*>(s_bias + kEpiWarps * N_TILE);
    uint32_t* s_misc = reinterpret_cast<uint32_t*>(s_bar + kNumBarriers);                  // tmem base, abort
    volatile uint32_t* s_abort = s_misc + 1;
    const uint32_t a_full0 = smem_u32(s_bar), a_empty0 = a_full0 + 8 * kMaxASlots, b_full0 = a_empty0 + 8 * kMaxASlots,
                   b_empty0 = b_full0 + 8 * kMaxBSlots, acc_full0 = b_empty0 + 8 * kMaxBSlots, acc_empty0 = acc_full0 + 16,
                   i_full0 = acc_empty0 + 16, i_empty0 = i_full0 + 8 * kIdxStages, sums0 = i_empty0 + 8 * kIdxStages, turn0 = sums0 + 32;

    const LutArgs& a = p.a;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rank = cluster_rank();
    const uint32_t n_items = p.tiles_m * p.tiles_n * (SPLIT ? p.split : 1u), n_pairs = gridDim.x >> 1, first = blockIdx.x >> 1;

    if (threadIdx.x == 0) {
        s_misc[1] = 0;
        tma_prefetch_desc(&lut_map);
        tma_prefetch_desc(&idx_map);
        tma_prefetch_desc(&out_map);
    }
    if (threadIdx.x >= 64 && threadIdx.x < 64 + kNumBarriers) {
        const uint32_t b = threadIdx.x - 64;
        // a_full: the four builder warps of the slab's group in each CTA; a_empty, b_empty: one commit; b_full: the
        // leader's expect_tx (the copies of both CTAs complete the bytes); acc_full: one commit per issuing warp;
        // acc_empty: the epilogue warps of both CTAs (barriers the
        // leader waits on are unused in the other CTA); i_full: expect_tx; i_empty: the CTA's builder warps;
        // four: a quadrant's partial sums are complete; the last kMmaWarps: an issuing warp's turn.
        const uint32_t after = 2 * kMaxASlots + 2 * kMaxBSlots;
        mbar_init(a_full0 + 8 * b, b < kMaxASlots ? 8u : b < after ? 1u : b < after + 2 ? kMmaWarps : b < after + 4 ? 2 * kEpiWarps : b < after + 4 + kIdxStages ? 1u : b < after + 4 + 2 * kIdxStages ? 4 * kGroups : 1u);
        fence_barrier_init();
    }
    if (warp == kFirstMma) tmem_alloc_pair(smem_u32(s_misc), 512);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(s_misc);
    const uint32_t my_lanes = ((warp & 3u) * 32u) << 16;
    if (warp >= kFirstEpi) {   // every MMA accumulates: the accumulators start at zero
        const uint32_t zero[32] = {}, used = p.one_tile ? N_TILE : accumulators(N_TILE) * N_TILE;
        for (uint32_t c = 0; c < used; c += 32) tmem_st_32x32b_x32(tmem_base + my_lanes + c, zero);
        tmem_st_wait();
    }
    tc_fence_before_sync();
    cluster_sync();   // barriers initialised and accumulators cleared in both CTAs
    tc_fence_after_sync();

    // The end of a tile, columns c * 32 and up, of a warp's lane quadrant.  v: 32 columns of this thread's row, into the
    // output through a staging block and the copy engine; bw: the block's bias values.
    auto finish = [&](const SparseItem& it, uint32_t c, const uint32_t (&v)[32], const float* bw, unsigned char* sg) {
        // straight-line code for all 32 columns: a branch per value leaves every latency of a lone warp exposed
        const float lbcb = lut_bias_times_cb(a.lut_bias, a.CB);
        float o[32];
#pragma unroll
        for (uint32_t q = 0; q < 8; ++q) {
            const float4 b4 = *reinterpret_cast<const float4*>(bw + 4 * q);
            o[4 * q] = dequant_one((int32_t)v[4 * q], a.scale, lbcb, b4.x);
            o[4 * q + 1] = dequant_one((int32_t)v[4 * q + 1], a.scale, lbcb, b4.y);
            o[4 * q + 2] = dequant_one((int32_t)v[4 * q + 2], a.scale, lbcb, b4.z);
            o[4 * q + 3] = dequant_one((int32_t)v[4 * q + 3], a.scale, lbcb, b4.w);
        }
        activate_all(o, a.act);
#pragma unroll
        for (uint32_t q = 0; q < 8; ++q)
            *reinterpret_cast<float4*>(sg + lane * 128 + ((q ^ (lane & 7u)) << 4)) = make_float4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
            tma_store_2d(&out_map, smem_u32(sg), (int32_t)(it.n0 + c * 32), (int32_t)(it.m0 + (warp & 3u) * 32));
            tma_store_commit();
        }
    };
    // One wide tile per pair: its end is nobody's to hide, so the builders, who are done, take their share of the
    // 32-column blocks, and as the slab ring is empty every block has a staging block there.  (In the narrower
    // instances the second copy of this code cost the main loop 5 % and more than the shorter end gave.)
    auto finish_one = [&](uint32_t helper) -> bool {
        const SparseItem it = sparse_item<SPLIT>(p, first, N_TILE, rank);
        const uint32_t quad = warp & 3u;
        float* bq = s_bias + quad * N_TILE;
        for (uint32_t c = helper; c < N_TILE / 32; c += 1 + kGroups) {
            const uint32_t n = it.n0 + c * 32 + lane;
            bq[c * 32 + lane] = n < a.N ? __ldg(a.bias + n) : 0.f;
        }
        uint32_t w_ok = 1;
        if (lane == 0) w_ok = mbar_wait<256>(acc_full0, 0, s_abort) ? 1u : 0u;
        if (!__shfl_sync(0xffffffffu, w_ok, 0)) return false;
        __syncwarp();   // all lanes' bias values, and what lane 0 waited for: a shuffle orders no memory
        tc_fence_after_sync();
        for (uint32_t c = helper; c < N_TILE / 32; c += 1 + kGroups) {
            if (it.n0 + c * 32 >= a.N || it.m0 + quad * 32 >= a.M) break;   // blocks wholly past N or M
            uint32_t v[32];
            tmem_ld_32x32b_x32(tmem_base + my_lanes + c * 32u, v);
            tmem_ld_wait();
            finish(it, c, v, bq + c * 32, s_b + (size_t)(quad * (N_TILE / 32) + c) * kStageBytes);
        }
        if (lane == 0) tma_store_wait_all();   // shared memory and the output are settled before the CTA leaves
        return true;
    };

    if (warp < kCopyWarps) {
        // ---------------- LUT copies (unless it was laid out just now the LUT does not depend on the preceding kernel),
        // slab x by warp x % kCopyWarps: a thread sustains one copy per ~ 480 cycles, of which the instruction itself
        // holds it for 350
        if (p.fresh_table) pdl_wait_prior_grid();
        if (lane == 0) {
            uint32_t j = warp, ph = 0, x0 = 0;
            bool ok = true;
            const uint32_t full_leader = map_to_rank(b_full0, 0);
            for (uint32_t item = first; item < n_items && ok; item += n_pairs) {
                const SparseItem it = sparse_item<SPLIT>(p, item, N_TILE, rank);
                for (uint32_t i = (warp - x0) & (kCopyWarps - 1); i < it.slabs; i += kCopyWarps) {
                    ok = mbar_wait<32>(b_empty0 + 8 * j, ph ^ 1, s_abort);
                    if (!ok) break;
                    if (rank == 0) mbar_arrive_expect_tx(b_full0 + 8 * j, 2 * kBBytes);
                    if constexpr (CANONICAL)
                        tma_load_4d_pair(smem_u32(s_b + (size_t)j * kBBytes), &lut_map, full_leader + 8 * j, (int32_t)(it.n0 + rank * kHalfN),
                                         (int32_t)((it.begin + i) * (kSlab >> LG)));
                    else
                        tma_load_3d_pair(smem_u32(s_b + (size_t)j * kBBytes), &lut_map, full_leader + 8 * j, 0,
                                         (int32_t)(it.n0 + rank * kHalfN), (int32_t)(2 * (it.begin + i)));
                    j += kCopyWarps;
                    if (j >= SB) { j -= SB; ph ^= 1; }
                }
                x0 += it.slabs;
            }
        }
        __syncwarp();
        if (p.early_trigger) pdl_launch_dependents();
    } else if (warp < kFirstMma) {
        // ---------------- index copies.  Straight loads by the builders, 16 bytes of a row each, were what a builder
        // waited for: beside the slabs an L2 access takes 1.5 us and more, and half of each sector was not used.
        pdl_wait_prior_grid();
        if (lane == 0) {
            uint32_t st = 0, ph = 0;
            bool ok = true;
            for (uint32_t item = first; item < n_items && ok; item += n_pairs) {
                const SparseItem it = sparse_item<SPLIT>(p, item, N_TILE, rank);
                for (uint32_t i = 0; i < it.slabs; i += kIdxSlabs) {
                    ok = mbar_wait<32>(i_empty0 + 8 * st, ph ^ 1, s_abort);
                    if (!ok) break;
                    mbar_arrive_expect_tx(i_full0 + 8 * st, kIdxBytes);
                    tma_load_2d(smem_u32(s_idx + st * kIdxBytes), &idx_map, i_full0 + 8 * st, (int32_t)((it.begin + i) * (kSlab >> LG)), (int32_t)it.m0);
                    if (++st == kIdxStages) { st = 0; ph ^= 1; }
                }
            }
        }
        __syncwarp();
        if (p.early_trigger) pdl_launch_dependents();
    } else if (warp < kFirstBuilder) {
        // ---------------- MMA issue, leader only: several warps, so that one is waiting when a slot fills.  All of them
        // accumulate into one accumulator, and that is ordered between instructions of one thread only; between threads it takes
        // the tcgen05 fences on either side of a barrier.  So the warps issue in turn, slab after slab, each
        // handing over behind its four instructions (not behind their completion).  Unordered, the four linears of BERT-base at
        // 1024 tokens take 76.4 us, in turn 76.8, 512 tokens 768 -> 3072 13.5 and 13.7, 65536 tokens 4096 -> 16384 12.46 and 12.68 ms; one
        // warp alone, which needs no hand-over, takes 81.8 and 15.1 us for the first two.  Converged loop, one elected lane issues.
        if (rank == 0) {
            const uint32_t me = warp - kFirstMma;
            uint32_t j = me, pb = 0, t = 0, x0 = 0;   // LUT slot and phases of this warp's next slab; slabs before the item
            bool ok = true;
            const uint64_t b_desc = CANONICAL ? umma_desc_columns(smem_u32(s_b), kHalfN) : umma_desc_k_sw128(smem_u32(s_b));
            const uint32_t b_lo0 = (uint32_t)b_desc, desc_hi = (uint32_t)(b_desc >> 32);
            // from one instruction's 64 positions to the next: two per 128-byte swizzle row, or 64 rows on
            constexpr uint32_t kOdd = CANONICAL ? 64 * kHalfN >> 4 : 4, kEven = CANONICAL ? 128 * kHalfN >> 4 : kHalfN * 128 >> 4;
            for (uint32_t item = first; item < n_items && ok; item += n_pairs, ++t) {
                const uint32_t ab = t & 1, slabs = sparse_item<SPLIT>(p, item, N_TILE, rank).slabs;
                ok = mbar_wait_warp(acc_empty0 + 8 * ab, ((t >> 1) & 1) ^ 1, s_abort);
                if (!ok) break;
                tc_fence_after_sync();
                const uint32_t d_tmem = tmem_base + ab * N_TILE;
                for (uint32_t i = (me - x0) & (kMmaWarps - 1); i < slabs; i += kMmaWarps) {
                    const uint32_t x = x0 + i, k = x % kASlots, pa = (x / kASlots) & 1u;
                    ok = mbar_wait(b_full0 + 8 * j, pb, s_abort) && mbar_wait(a_full0 + 8 * k, pa, s_abort) &&
                         mbar_wait(turn0 + 8 * me, ((x / kMmaWarps) & 1u) ^ (me == 0 ? 1u : 0u), s_abort);   // slab 0 has its turn
                    tc_fence_after_sync();
                    if (elect_one()) {
                        const uint32_t b_lo = b_lo0 + j * (kBBytes >> 4);
#pragma unroll
                        for (uint32_t kk = 0; kk < 4; ++kk)
                            umma_i8_sparse_pair(d_tmem, tmem_base + kDataBase + 32 * k + 8 * kk,
                                                ((uint64_t)desc_hi << 32) | (b_lo + (kk >> 1) * kEven + (kk & 1) * kOdd),
                                                tmem_base + kMetaBase + 2 * k, kIdesc);
                        tc_fence_before_sync();
                        mbar_arrive(turn0 + 8 * ((me + 1) & (kMmaWarps - 1)));
                        umma_commit_pair(a_empty0 + 8 * k);
                        umma_commit_pair(b_empty0 + 8 * j);
                    }
                    ok = __all_sync(0xFFFFFFFFu, ok);   // behind the instructions: see ptx.cuh
                    if (!ok) break;
                    j += kMmaWarps;
                    if (j >= SB) { j -= SB; pb ^= 1; }
                }
                x0 += slabs;
                if (ok && elect_one()) umma_commit_pair(acc_full0 + 8 * ab);
                __syncwarp();
            }
        }
        __syncwarp();
        if (p.early_trigger) pdl_launch_dependents();
    } else if (warp < kFirstEpi) {
        // ---------------- operand builders: slab x of the CTA's sequence by group x % 4, into slot x % kASlots
        constexpr int kRaw = LG == 3 ? 8 : 4;
        const uint32_t grp = (warp - kFirstBuilder) >> 2, r = (warp & 3u) * 32 + lane;
        // the 256 / CT index bytes of slab `sub` of a stage; 64-byte rows are swizzled
        auto load_raw = [&](const unsigned char* st, uint32_t sub, uint32_t (&v)[kRaw]) {
            const unsigned char* row = st + r * kIdxWidth;
            if constexpr (LG == 3) {
                const uint4 t = *reinterpret_cast<const uint4*>(row + (((2 * sub) ^ ((r >> 1) & 3u)) << 4));
                const uint4 u = *reinterpret_cast<const uint4*>(row + (((2 * sub + 1) ^ ((r >> 1) & 3u)) << 4));
                v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w; v[4] = u.x; v[5] = u.y; v[6] = u.z; v[7] = u.w;
            } else if constexpr (LG == 4) {
                const uint4 t = *reinterpret_cast<const uint4*>(row + ((sub ^ ((r >> 1) & 3u)) << 4));
                v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
            } else if constexpr (LG == 5) {
                const uint2 t = *reinterpret_cast<const uint2*>(row + 8 * sub);
                v[0] = t.x; v[1] = t.y;
            } else if constexpr (LG == 6) {
                v[0] = *reinterpret_cast<const uint32_t*>(row + 4 * sub);
            } else if constexpr (LG == 7) {
                v[0] = *reinterpret_cast<const uint16_t*>(row + 2 * sub);
            } else {
                v[0] = row[sub];
            }
        };
        const uint32_t full_leader = map_to_rank(a_full0, 0);
        uint32_t x0 = 0, st = 0, ph = 0;
        bool ok = true;
        for (uint32_t item = first; item < n_items && ok; item += n_pairs) {
            const uint32_t slabs = sparse_item<SPLIT>(p, item, N_TILE, rank).slabs;
            for (uint32_t i0 = 0; i0 < slabs && ok; i0 += kIdxSlabs) {
                ok = mbar_wait(i_full0 + 8 * st, ph, s_abort);
                for (uint32_t i = (grp - (x0 + i0)) & (kGroups - 1); i < kIdxSlabs && i0 + i < slabs; i += kGroups) {
                    const uint32_t x = x0 + i0 + i, k = x % kASlots, pa = (x / kASlots) & 1u;
                    uint32_t raw[kRaw], w[32], m[2];
                    load_raw(s_idx + st * kIdxBytes, i, raw);
                    build_row<LG, CANONICAL ? LG - 1 : 1>(raw, w, m);
                    // the row is in registers before the slot is waited for (the compiler would sink it behind the wait,
                    // onto the slot's turn-around path)
#pragma unroll
                    for (int c = 0; c < 32; ++c) asm volatile("" : "+r"(w[c]));
                    asm volatile("" : "+r"(m[0]), "+r"(m[1]));
                    ok = mbar_wait(a_empty0 + 8 * k, pa ^ 1, s_abort) && ok;
                    tc_fence_after_sync();
                    tmem_st_32x32b_x32(tmem_base + my_lanes + kDataBase + 32 * k, w);
                    tmem_st_32x32b_x2(tmem_base + my_lanes + kMetaBase + 2 * k, m);
                    tmem_st_wait();
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(full_leader + 8 * k);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(i_empty0 + 8 * st);   // this warp has read its rows of the stage
                ok = __all_sync(0xFFFFFFFFu, ok);
                if (++st == kIdxStages) { st = 0; ph ^= 1; }
            }
            x0 += slabs;
        }
        if (p.early_trigger) pdl_launch_dependents();
        if constexpr (SPLIT) {
            pdl_wait_prior_grid();
            if (ok && first < n_items) split_finish<N_TILE>(p, sparse_item<SPLIT>(p, first, N_TILE, rank), rank, warp & 3u, 1 + grp, lane, sums0, s_abort);
        } else if constexpr (kOne) {
            pdl_wait_prior_grid();
            if (ok && first < n_items) finish_one(1 + grp);
        }
        __syncwarp();
        tc_fence_before_sync();
    } else {
        // ---------------- epilogue: each warp on the lane quadrant it may read
        pdl_wait_prior_grid();
        const uint32_t quad = warp & 3u;
        unsigned char* stg = s_stage + (warp - kFirstEpi) * (kStages * kStageBytes);
        float* bw = s_bias + (warp - kFirstEpi) * N_TILE;
        const uint32_t empty_leader = map_to_rank(acc_empty0, 0);
        uint32_t t = 0, buf = 0;
        bool ok = true;
        if constexpr (kOne) {
            if (p.early_trigger) pdl_launch_dependents();
            if (first < n_items) finish_one(0);
        }
        for (uint32_t item = first; item < n_items && !kOne; item += n_pairs, ++t) {
            const SparseItem it = sparse_item<SPLIT>(p, item, N_TILE, rank);
            const uint32_t ab = t & 1;
            if (p.early_trigger && item + n_pairs >= n_items) pdl_launch_dependents();
            __syncwarp();   // the previous item's reads of bw are done
#pragma unroll
            for (uint32_t c = 0; c < N_TILE / 32; ++c) {
                const uint32_t n = it.n0 + c * 32 + lane;
                bw[c * 32 + lane] = n < a.N ? __ldg(a.bias + n) : 0.f;
            }
            uint32_t w_ok = 1;
            if (lane == 0) w_ok = (ok && mbar_wait<256>(acc_full0 + 8 * ab, (t >> 1) & 1, s_abort)) ? 1u : 0u;
            ok = __shfl_sync(0xffffffffu, w_ok, 0) != 0;
            if (!ok) continue;
            __syncwarp();   // all lanes' bias values, and what lane 0 waited for: a shuffle orders no memory
            tc_fence_after_sync();
            constexpr uint32_t kChunks = N_TILE / 32;
            const uint32_t corner = (it.tile * 2 + rank) * 4 + quad;
            for (uint32_t c = 0; c < kChunks; ++c) {
                uint32_t v[32];
                tmem_ld_32x32b_x32(tmem_base + my_lanes + ab * N_TILE + c * 32u, v);
                tmem_ld_wait();
                {   // leave the columns at zero for the next item's accumulating MMAs
                    const uint32_t zero[32] = {};
                    tmem_st_32x32b_x32(tmem_base + my_lanes + ab * N_TILE + c * 32u, zero);
                }
                if (c == kChunks - 1) {   // accumulator fully read and cleared: hand the buffer back
                    tmem_st_wait();
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(empty_leader + 8 * ab);
                }
                if constexpr (!SPLIT) {
                    if (it.n0 + c * 32 < a.N && it.m0 + quad * 32 < a.M) {   // not wholly past N or M
                        if (lane == 0) tma_store_wait_read_1();   // the copy before last has read this buffer
                        __syncwarp();
                        finish(it, c, v, bw + c * 32, stg + buf * kStageBytes);
                        buf ^= 1;
                    }
                } else {
                    uint4* to = partial_sums<N_TILE>(p, corner, it.z, c, lane);
#pragma unroll
                    for (uint32_t q = 0; q < 8; ++q) __stcg(to + 32 * q, make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]));
                }
            }
            if constexpr (SPLIT) {
                __threadfence();
                __syncwarp();
                if (lane == 0) atomicAdd(p.counters + 2 * corner, 1u);
                ok = split_finish<N_TILE>(p, it, rank, quad, 0, lane, sums0, s_abort);
            }
        }
        if (lane == 0) tma_store_wait_all();   // shared memory and the output are settled before the CTA leaves
        __syncwarp();
        tc_fence_before_sync();
    }

    // ---------------- tear-down (also the way out after a wait that ran out)
    __syncthreads();
    if (*s_abort) {
        if (threadIdx.x == 0) {
            // give copies that may still be in flight a bounded time to land before the shared memory is handed back
            const long long t0 = clock64();
            while (clock64() - t0 < 200000) {}
            report_error(p.dev_err, 2u);
        }
        __syncthreads();
    }
    cluster_sync();   // nothing of this CTA is read, written or signalled by the other one any more
    if (warp == kFirstMma) {
        tc_fence_after_sync();
        tmem_dealloc_pair(tmem_base, 512);
    }
}

constexpr size_t kSmemLimit = 227 * 1024;

uint32_t log2_of(uint32_t v) {
    uint32_t lg = 0;
    while ((1u << lg) < v) ++lg;
    return lg;
}
uint32_t sparse_slabs(uint32_t CB, uint32_t CT) { return (uint32_t)(((uint64_t)CB * CT + kSlab - 1) / kSlab); }

size_t sparse_smem(uint32_t n_tile, int lg, uint32_t b_slots) {
    return (size_t)b_slots * (n_tile / 2) * kSlab + stage_blocks(n_tile) * kStageBytes + kIdxStages * kRows * idx_width(lg) +
           kEpiWarps * n_tile * 4 + kNumBarriers * 8 + 16 + 1024;
}

template <uint32_t N_TILE, int LG, bool SPLIT, bool CANONICAL>
cudaError_t run(const CUtensorMap& map, const CUtensorMap& idx_map, const CUtensorMap& out_map, const SparseParams& p, uint32_t pairs, size_t smem, cudaStream_t s) {
    auto k = lut_sparse_kernel<N_TILE, LG, SPLIT, CANONICAL>;
    static SmemOptIn memo;
    cudaError_t e = allow_smem(memo, k, (int)smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * pairs);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, k, map, idx_map, out_map, p);
}

template <uint32_t N_TILE, bool SPLIT, bool CANONICAL = false>
cudaError_t run_lg(uint32_t lg, const CUtensorMap& map, const CUtensorMap& idx_map, const CUtensorMap& out_map, const SparseParams& p, uint32_t pairs, size_t smem, cudaStream_t s) {
    switch (lg) {
        case 3: return run<N_TILE, 3, SPLIT, CANONICAL>(map, idx_map, out_map, p, pairs, smem, s);
        case 4: return run<N_TILE, 4, SPLIT, CANONICAL>(map, idx_map, out_map, p, pairs, smem, s);
        case 5: return run<N_TILE, 5, SPLIT, CANONICAL>(map, idx_map, out_map, p, pairs, smem, s);
        case 6: return run<N_TILE, 6, SPLIT, CANONICAL>(map, idx_map, out_map, p, pairs, smem, s);
        case 7: return run<N_TILE, 7, SPLIT, CANONICAL>(map, idx_map, out_map, p, pairs, smem, s);
        default: return run<N_TILE, 8, SPLIT, CANONICAL>(map, idx_map, out_map, p, pairs, smem, s);
    }
}

}  // namespace

uint32_t sparse_table_ctas(uint32_t CB, uint32_t CT, uint32_t N) { return sparse_slabs(CB, CT) * ((N + 63) / 64); }
size_t sparse_table_bytes(uint32_t CB, uint32_t CT, uint32_t N) { return (size_t)sparse_slabs(CB, CT) * kSlab * N; }

// The table as the kernel above wants it: [N][slabs * 256], row n's slab s holding at position 2 (d * codebooks + c) + h
// the entry of codebook s * codebooks + c and centroid index (d without its bit 1, h = bit 1); positions of codebooks
// past the last one are zero.  A block turns 256 rows x 64 columns of the canonical table: a thread takes the four rows
// that make one word of the result, four columns of each, and turns the 4 x 4 bytes in registers.
//
// What bounds it: the latency of one round of loads, so all 16 of a thread are in flight together (one after another
// a 1024-column table of 384 codebooks took 12 us; the call that lays out three of them in a row 88 -> 53 us).  In a chain of tables and contractions through the same memory
// (`chained`: the canonical table was complete before the kernel in front began) they are issued while that one still
// runs, on the SMs it leaves idle; the stores wait for it.
namespace {
__global__ void __launch_bounds__(256) sparse_table_kernel(const int8_t* __restrict__ lut, int8_t* __restrict__ out, uint32_t rows, uint32_t N,
                                                           uint32_t first, uint32_t pitch, uint32_t lg, uint32_t slabs, bool chained) {
    constexpr uint32_t kPitch = 65;   // words
    __shared__ uint32_t tile[64 * kPitch];
    pdl_launch_dependents();
    if (!chained) pdl_wait_prior_grid();
    const uint32_t slab = blockIdx.x, n0 = blockIdx.y * 64, lg_cbs = 8 - lg, n = (threadIdx.x & 15u) * 4, w0 = threadIdx.x >> 4;
    uint32_t v[4][4];
#pragma unroll
    for (uint32_t u = 0; u < 4; ++u) {
#pragma unroll
        for (uint32_t b = 0; b < 4; ++b) {
            const uint32_t pos = 4 * (w0 + 16 * u) + b, d = (pos >> 1) >> lg_cbs, c = (pos >> 1) & ((1u << lg_cbs) - 1u);
            const uint32_t row = slab * 256 + (c << lg) + ((d >> 1) << 2 | (pos & 1u) << 1 | (d & 1u));
            v[u][b] = 0;
            if (row < rows && n0 + n < N) v[u][b] = *reinterpret_cast<const uint32_t*>(lut + (size_t)row * pitch + first + n0 + n);   // columns in multiples of 16
        }
    }
#pragma unroll
    for (uint32_t u = 0; u < 4; ++u) {
        const uint32_t l0 = __byte_perm(v[u][0], v[u][1], 0x5140), l1 = __byte_perm(v[u][2], v[u][3], 0x5140);
        const uint32_t h0 = __byte_perm(v[u][0], v[u][1], 0x7362), h1 = __byte_perm(v[u][2], v[u][3], 0x7362);
        uint32_t* t = tile + n * kPitch + w0 + 16 * u;
        t[0] = __byte_perm(l0, l1, 0x5410); t[kPitch] = __byte_perm(l0, l1, 0x7632);
        t[2 * kPitch] = __byte_perm(h0, h1, 0x5410); t[3 * kPitch] = __byte_perm(h0, h1, 0x7632);
    }
    __syncthreads();
    if (chained) pdl_wait_prior_grid();
#pragma unroll
    for (uint32_t k = 0; k < 16; ++k) {
        const uint32_t r = (threadIdx.x >> 6) + 4 * k, w = threadIdx.x & 63u;
        if (n0 + r < N) *reinterpret_cast<uint32_t*>(out + ((size_t)(n0 + r) * slabs + slab) * 256 + 4 * w) = tile[r * kPitch + w];
    }
}
}  // namespace

cudaError_t launch_sparse_table(const int8_t* lut, int8_t* out, uint32_t CB, uint32_t CT, uint32_t N, uint32_t n0, uint32_t pitch, bool chained, cudaStream_t s) {
    const uint32_t slabs = sparse_slabs(CB, CT);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(slabs, (N + 63) / 64);
    cfg.blockDim = dim3(256);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, sparse_table_kernel, lut, out, CB * CT, N, n0, pitch, log2_of(CT), slabs, chained);
}

// That table as boxes of half a tile's rows of one slab: x = position within 128, y = row, z = half slab.
cudaError_t sparse_make_tmap(CUtensorMap* out, const int8_t* table, uint32_t CB, uint32_t CT, uint32_t N, uint32_t n_tile, const char** why) {
    *why = nullptr;
    EncodeTiledFn enc = get_encode_tiled();
    if (!enc) { *why = "cuTensorMapEncodeTiled is not available from this driver"; return cudaErrorNotSupported; }
    const uint64_t row = (uint64_t)sparse_slabs(CB, CT) * kSlab;
    cuuint64_t dims[3] = {128, N, row / 128};
    cuuint64_t strides[2] = {row, 128};
    cuuint32_t box[3] = {128, n_tile / 2, 2};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<int8_t*>(table), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { *why = "cuTensorMapEncodeTiled failed for the LUT slab map"; return cudaErrorInvalidValue; }
    return cudaSuccess;
}

// The canonical table [CB][CT][N] as boxes of half a tile's columns of one slab's 256 rows, in the order of the slab's
// positions 2 (d * codebooks + c) + h: columns, h (the highest bit of the centroid index), codebook, d (the bits below).
cudaError_t sparse_make_canonical_tmap(CUtensorMap* out, const int8_t* lut, uint32_t CB, uint32_t CT, uint32_t N, uint32_t n_tile, const char** why) {
    *why = nullptr;
    EncodeTiledFn enc = get_encode_tiled();
    if (!enc) { *why = "cuTensorMapEncodeTiled is not available from this driver"; return cudaErrorNotSupported; }
    cuuint64_t dims[4] = {N, 2, CB, CT / 2};
    cuuint64_t strides[3] = {(cuuint64_t)CT / 2 * N, (cuuint64_t)CT * N, N};
    cuuint32_t box[4] = {n_tile / 2, 2, kSlab / CT, CT / 2};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<int8_t*>(lut), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     n_tile == 64 ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { *why = "cuTensorMapEncodeTiled failed for the canonical table"; return cudaErrorInvalidValue; }
    return cudaSuccess;
}

// uint8 indices [M][CB] as 128 rows x idx_width bytes
cudaError_t sparse_make_idx_tmap(CUtensorMap* out, const uint8_t* idx, uint32_t M, uint32_t CB, uint32_t CT, const char** why) {
    *why = nullptr;
    EncodeTiledFn enc = get_encode_tiled();
    if (!enc) { *why = "cuTensorMapEncodeTiled is not available from this driver"; return cudaErrorNotSupported; }
    const uint32_t width = idx_width(log2_of(CT));
    cuuint64_t dims[2] = {CB, M};
    cuuint64_t strides[1] = {CB};
    cuuint32_t box[2] = {width, kRows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t*>(idx), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     width == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { *why = "cuTensorMapEncodeTiled failed for the index map (is the index buffer 16-byte aligned?)"; return cudaErrorInvalidValue; }
    return cudaSuccess;
}

// slabs whose index bytes fill the 16 bytes a copy must start on: a slice begins at a multiple
static uint32_t slice_unit(uint32_t CT) { return CT > 16 ? CT / 16 : 1; }

// Tile width and split of the codebook axis by the time the launch would take.  Rounds of one tile per pair, each bound by
// its slabs or, where the codebook axis is short, by the epilogue beside them (0.93 us per 32 columns), and the last
// tile's epilogue.  A slab takes 170 / 199 / 220 ns at 64 / 128 / 160 columns: at 64 the chain of one slot's
// turn-around, at 160 close to the tensor pipe's 320 cycles.  192 columns only where they make one round of what would be
// two: 384 codebooks of 16 -> 3072 at 1024 tokens 15.8 -> 12.7 us, 1024 codebooks 29.6 -> 21.3 (four LUT slots instead of
// eight at 256 columns: 27.8 and 15.4).  (Measured at 32 to 16384 tokens; at 96 columns nothing gained.)  Where the tiles leave pairs idle the axis is split over them, one item per pair, which costs 5 to 6 us for the
// partial sums' way through L2 (1536 codebooks -> 768 at 128 tokens 20.7 -> 12.2 us, at 1024 tokens 21.6 -> 17.6).
// only: the one tile width to choose the split for, 0 = any; most_split: 1 for a caller that has no scratch.
float sparse_default_plan(uint32_t M, uint32_t CB, uint32_t CT, uint32_t N, int sm_count, uint32_t* n_tile, uint32_t* split, uint32_t only, uint32_t most_split) {
    const uint32_t pairs = sm_count >= 2 ? (uint32_t)sm_count / 2 : 1, slabs = sparse_slabs(CB, CT), unit = slice_unit(CT);
    const uint64_t tm = (M + 2 * kRows - 1) / (2 * kRows);
    const struct { uint32_t n; float slab_us, split_us; } tiles[] = {{64, 0.170f, 5.f}, {128, 0.199f, 6.2f}, {160, 0.220f, 0.f}, {192, 0.250f, 0.f}};
    *n_tile = only ? only : 160;
    *split = 1;
    float least = 3e38f;
    for (const auto& t : tiles) {
        const uint64_t items = tm * ((N + t.n - 1) / t.n), rounds = (items + pairs - 1) / pairs;
        if (only ? t.n != only : accumulators(t.n) == 1 && rounds > 1) continue;
        const uint32_t most = items < pairs ? (uint32_t)(pairs / items) : 1;
        for (uint32_t s = 1; s <= most && s <= (t.n >= 160 ? 1u : most_split) && (s == 1 || s * unit <= slabs); ++s) {
            const uint32_t per = ((slabs + s - 1) / s + unit - 1) / unit * unit;
            const float main = per * t.slab_us, epi = 0.93f * (t.n / 32);
            const float us = (float)rounds * (rounds > 1 && epi > main ? epi : main) + 0.25f * (t.n / 32) + (s > 1 ? t.split_us : 0.f);
            if (us < least) { least = us; *n_tile = t.n; *split = (slabs + per - 1) / per; }
        }
    }
    return least;
}

// Tiles a plan may name; 192 columns suit only launches of one round, which sparse_default_plan() knows.
bool sparse_tile_ok(uint32_t n_tile) { return n_tile == 64 || n_tile == 128 || n_tile == 160; }

// The same for the canonical table: its tile width, and the time.  A slab takes what it takes above where the rows that
// the copies fetch, 64 or 32 bytes of 256 table rows, begin on multiples of 64 or 32 bytes, and up to twice that where
// N makes every other one straddle sectors (2048 codebooks of 16, 64 tokens: N = 3136 44 us a call in 128-wide tiles, 3104 56,
// 3088 73, in 64-wide ones 57).
float sparse_canonical_plan(uint32_t M, uint32_t CB, uint32_t CT, uint32_t N, int sm_count, uint32_t* n_tile) {
    const uint32_t pairs = sm_count >= 2 ? (uint32_t)sm_count / 2 : 1, slabs = sparse_slabs(CB, CT);
    const uint64_t tm = (M + 2 * kRows - 1) / (2 * kRows);
    const struct { uint32_t n; float slab_us; } tiles[] = {{64, N % 32 ? 0.29f : 0.17f}, {128, N % 32 ? 0.42f : N % 64 ? 0.27f : 0.2f}};
    float least = 3e38f;
    for (const auto& t : tiles) {
        const uint64_t rounds = (tm * ((N + t.n - 1) / t.n) + pairs - 1) / pairs;
        const float main = slabs * t.slab_us, epi = 0.93f * (t.n / 32), us = (float)rounds * (rounds > 1 && epi > main ? epi : main) + 0.25f * (t.n / 32);
        if (us < least) { least = us; *n_tile = t.n; }
    }
    return least;
}

// Scratch of a split launch: partial sums and counter words.
void sparse_split_scratch(uint32_t M, uint32_t N, uint32_t n_tile, uint32_t split, size_t* partial_bytes, size_t* counter_bytes) {
    const size_t tiles = (size_t)((M + 2 * kRows - 1) / (2 * kRows)) * ((N + n_tile - 1) / n_tile);
    *partial_bytes = split > 1 ? tiles * split * 2 * kRows * n_tile * sizeof(int32_t) : 0;
    *counter_bytes = split > 1 ? tiles * 8 * 2 * sizeof(uint32_t) : 0;
}

cudaError_t launch_sparse(const LutArgs& a, const CUtensorMap& lut_map, const CUtensorMap& idx_map, const CUtensorMap& out_map, uint32_t n_tile,
                          uint32_t split, void* partial, uint32_t* counters, uint32_t max_ctas, bool fresh_table, bool canonical, uint32_t* dev_err,
                          cudaStream_t s, const char** why) {
    *why = nullptr;
    if (a.M == 0 || a.N == 0) return cudaSuccess;
    SparseParams p;
    p.a = a;
    p.slabs = sparse_slabs(a.CB, a.CT);
    p.tiles_m = (a.M + 2 * kRows - 1) / (2 * kRows);
    p.tiles_n = (a.N + n_tile - 1) / n_tile;
    const uint32_t cap = max_ctas / 2, unit = slice_unit(a.CT);
    // the slices of a tile wait for one another: only where every item has a pair of its own
    if (!split || n_tile >= 160 || (uint64_t)p.tiles_m * p.tiles_n * split > cap || !partial || !counters) split = 1;
    p.per = ((p.slabs + split - 1) / split + unit - 1) / unit * unit;
    p.split = (p.slabs + p.per - 1) / p.per;   // no empty slices
    p.partial = static_cast<uint4*>(partial);
    p.counters = counters;
    p.dev_err = dev_err;
    const int lg = (int)log2_of(a.CT);
    p.b_slots = kMaxBSlots;   // a multiple of the issuing warps: every slot has one of them
    while (p.b_slots > kMmaWarps && sparse_smem(n_tile, lg, p.b_slots) > kSmemLimit) p.b_slots -= kMmaWarps;
    const uint64_t items = (uint64_t)p.tiles_m * p.tiles_n * p.split;
    const uint32_t pairs = (uint32_t)(items < cap ? items : cap);
    // All pairs work on the same columns at a time and share their slabs in L2.  Where the indices of all rows would not
    // stay there from one column tile to the next (65536 tokens x 2048 codebooks: 134 MB, read from memory 103 times),
    // go through the columns with as many row tiles as there are pairs: 13.8 GB of reads become 1.9 GB of table.
    p.group_m = (uint64_t)a.M * a.CB > (48ull << 20) && p.tiles_m > cap ? cap : p.tiles_m;
    p.one_tile = items <= cap;
    // With one tile per pair all pairs reach the end of their main loops together, and the next kernel of the stream may as
    // well be launched then; with several they finish a tile apart and its early CTAs would skew it.  Where they go are the SMs
    // that the tiles leave idle, as many to an SM as fit: that pays where the next kernel is a light search of up to four
    // CTAs per idle SM, or the layout of the next piece of a table (256 threads and 16 loads each) of up to eight.  Measured
    // on chains of an encoder layer's four linears, without the trigger / always with it: width 768, v = 2, 16 centroids at 128 tokens 48.7 / 50.7 us,
    // by this rule 49.3; v = 4 at 128 41.7 / 43.6 / 41.0; 32 centroids at 512 90 / 102 / 90; v = 4, 64 centroids at 320 104 / 123 / 104;
    // width 1280, v = 4 at 64 54.7 / 50.7 / 50.5; 1024, v = 4 at 384 60.2 / 56.9 / 58.0, at 32 (rows) 36.9 / 42.4 / 36.9.
    // Tables in pieces (never / always): 768 -> 3072 at 512 tokens (4.6 CTAs per idle SM) 53.4 / 50.7 us, at 1024 (19) 55.0 / 59.2; 512 ->
    // 8192 at 640 (5.9) 76.9 / 73.3, at 384 (9.5) 72.6 / 80.7.
    p.early_trigger = p.one_tile && a.next_ctas && a.next_ctas <= a.next_per_sm * (max_ctas - 2 * pairs);
    p.fresh_table = fresh_table;
    if (accumulators(n_tile) == 1 && !p.one_tile) { *why = "tiles wider than 160 columns of the sparse form take one tile per pair"; return cudaErrorInvalidValue; }
    const size_t smem = sparse_smem(n_tile, lg, p.b_slots);
    if (canonical) {
        if (p.split == 1 && n_tile == 64) return run_lg<64, false, true>(lg, lut_map, idx_map, out_map, p, pairs, smem, s);
        if (p.split == 1 && n_tile == 128) return run_lg<128, false, true>(lg, lut_map, idx_map, out_map, p, pairs, smem, s);
        *why = "the canonical table is contracted in 64- and 128-wide tiles, unsplit";
        return cudaErrorInvalidValue;
    }
#define LUTAMM_SPARSE_CASE(NT, SP) \
    if (n_tile == NT && (p.split > 1) == SP) return run_lg<NT, SP>(lg, lut_map, idx_map, out_map, p, pairs, smem, s);
    LUTAMM_SPARSE_CASE(64, false)
    LUTAMM_SPARSE_CASE(64, true)
    LUTAMM_SPARSE_CASE(128, false)
    LUTAMM_SPARSE_CASE(128, true)
    LUTAMM_SPARSE_CASE(160, false)
    LUTAMM_SPARSE_CASE(192, false)
#undef LUTAMM_SPARSE_CASE
    *why = "tcgen05 variant: the sparse form is built for 64-, 128-, 160- and (one tile per pair) 192-wide tiles";
    return cudaErrorInvalidValue;
}

}  // namespace lutamm
