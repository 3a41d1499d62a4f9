// Internal launcher interface between the C ABI (lutamm_capi.cu) and the kernels.
#pragma once
#include <atomic>
#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>

namespace lutamm {

// ---- step 1: closest-centroid search -------------------------------------------------
struct CcsArgs {
    const float* x;         // [M][K]
    const float* centroid;  // [CB][CT][v]
    void* idx_out;          // uint8 [M][CB] or uint16 tiled
    uint32_t M, K, v, CB, CT;
    uint32_t format;        // LUTAMM_INDEX_*
    uint32_t n_stile, cb_mtile;  // tiled format only
    uint32_t tokens_per_thread;  // 0 = default
    uint32_t* dev_err;           // null: without the form on the tensor cores, which has waits that may run out
};
cudaError_t launch_ccs(const CcsArgs& a, cudaStream_t s, const char** why);
// ... on the tensor cores, for many tokens (ccs_umma.cu), and the calls it can take
bool ccs_umma_takes(const CcsArgs& a);
cudaError_t launch_ccs_umma(const CcsArgs& a, cudaStream_t s);
bool ccs_reads_tokens_per_thread(uint32_t v, uint32_t CT);
bool ccs_has_short_form(uint32_t v, uint32_t CT);   // for small calls
// CTAs of the search in its short form, where their centroids are at most 64 floats a codebook: such CTAs do as well
// several to an SM as spread out.  0 where the search has another form.
uint32_t ccs_light_ctas(uint32_t M, uint32_t CB, uint32_t CT, uint32_t v);

// ---- step 2+3: gather-accumulate + dequantise -----------------------------------------
// Output addressing: row-major [M][N], or the reference's DPU-tiled layout.
struct OutLayout {
    uint32_t tiled;  // 0 = row-major
    uint32_t n_stile, f_stile, f_mtile, lut_par;
};

struct LutArgs {
    const uint8_t* idx;   // [M][CB]
    const float* bias;    // [N]
    float* out;           // fp32, layout per `layout`
    int32_t* acc_out;     // optional int32 [M][N] row-major (parity checks), may be null
    uint32_t M, CB, CT, N;
    float scale, lut_bias;
    OutLayout layout;
    uint32_t act;         // LUTAMM_ACT_*: applied after the dequantisation
    uint32_t next_ctas, next_per_sm;  // CTAs of the kernel that is expected next in the stream (0: not known, or not to be
                                      // launched early), and how many of them an SM without a tile takes well
    // Column sharding with the exchange fused into the kernel: the [M][N] block is also stored, by plain
    // st.global over NVLink, at the same offsets of n_peers - 1 other GPUs' buffers (peer_out[g] points at
    // this rank's block inside GPU g's gathered buffer; the entry for this GPU itself equals `out` and is
    // skipped).  n_peers == 0: a purely local store.  tcgen05 variant, row-major output only.
    uint32_t n_peers;
    float* peer_out[8];
};
constexpr uint32_t kMaxPeers = 8;

// Gather variant: LUT canonical [CB][CT][N] staged by 3-D TMA tiles.
struct GatherPlan {
    uint32_t cfg;  // tile configuration id
};
uint32_t gather_num_cfgs();
// microseconds a launch takes
float gather_us(uint32_t M, uint32_t CB, uint32_t CT, uint32_t N, uint32_t cfg, int sm_count);
// Encodes the tensor map the configuration needs (box sizes depend on it).
cudaError_t gather_make_tmap(CUtensorMap* out, const int8_t* lut, uint32_t CB, uint32_t CT, uint32_t N, uint32_t cfg,
                             const char** why);
cudaError_t launch_gather(const LutArgs& a, const CUtensorMap& lut_map, uint32_t cfg, uint32_t* dev_err,
                          cudaStream_t s, const char** why);

// tcgen05 variant: LUT transposed to K-major [N][CB*CT] at load time, 2-D TMA tiles with
// 128-byte swizzle; the one-hot operand is synthesised in shared memory from the indices.
struct UmmaPlan {
    uint32_t n_tile;    // 64 / 128 / 256 (A in shared memory), 64 / 128 / 192 (A in tensor memory)
    uint32_t a_tmem;    // 1: the one-hot operand is written to tensor memory instead of shared memory
    uint32_t split;     // work items sharing one output tile along the codebook axis
    uint32_t stages;    // LUT slabs in flight in shared memory (0 = as many as fit)
    uint32_t groups;    // one-hot builder groups of four warps (0 = default)
    uint32_t sps;       // 128-byte slabs a one-hot builder group takes per turn: 1 or 2 (0 = by ring depth)
    uint32_t max_ctas;  // persistent grid size cap: the SM count
    uint32_t epilogue;  // 1 = transposing stores; 0 / 2 = tiled bulk stores where the launch admits them
};
bool umma_supported(uint32_t CB, uint32_t CT, uint32_t N);
bool umma_tile_ok(uint32_t n_tile, bool a_tmem);
cudaError_t umma_make_tmap(CUtensorMap* out, const int8_t* lut_t, uint32_t CB, uint32_t CT, uint32_t N,
                           uint32_t n_tile, const char** why);
// `acc_scratch` (int32 [split][M][N]) and `tile_counters` (two words per output tile, zeroed once)
// are needed when split > 1.
cudaError_t launch_umma(const LutArgs& a, const CUtensorMap& lut_t_map, const UmmaPlan& p, int32_t* acc_scratch,
                        uint32_t* tile_counters, uint32_t* dev_err, cudaStream_t s, const char** why);
void umma_default_plan(uint32_t M, uint32_t CB, uint32_t CT, uint32_t N, int sm_count, uint32_t operand,
                       uint32_t n_tile, uint32_t sps, UmmaPlan* p);
uint32_t umma_auto_split(uint32_t M, uint32_t CB, uint32_t CT, uint32_t N, uint32_t n_tile, int sm_count);

// fp32 [M][N] row-major output as 32 x 32 blocks with the 128-byte swizzle the epilogues stage them in
// (`pitch`: floats from row to row, 0 = N)
cudaError_t make_out_tmap(CUtensorMap* out, float* base, uint32_t M, uint32_t N, const char** why, uint32_t pitch = 0);

// The same contraction on CTA pairs with the one-hot operand 2:4 sparse (row-major fp32 output): from its own layout of
// the table (sparse_table_bytes of it), at twice the rate.
size_t sparse_table_bytes(uint32_t CB, uint32_t CT, uint32_t N);
uint32_t sparse_table_ctas(uint32_t CB, uint32_t CT, uint32_t N);
// ... of `n` columns of a table that has `pitch`, from column n0 on; chained: nothing the stream still runs writes `lut`
cudaError_t launch_sparse_table(const int8_t* lut, int8_t* out, uint32_t CB, uint32_t CT, uint32_t n, uint32_t n0, uint32_t pitch, bool chained, cudaStream_t s);
// Tile width (`only`, where that is not 0) and split (up to most_split); returns the microseconds it expects, launch apart
// (about 4)
float sparse_default_plan(uint32_t M, uint32_t CB, uint32_t CT, uint32_t N, int sm_count, uint32_t* n_tile, uint32_t* split, uint32_t only = 0,
                          uint32_t most_split = 16);
void sparse_split_scratch(uint32_t M, uint32_t N, uint32_t n_tile, uint32_t split, size_t* partial_bytes, size_t* counter_bytes);
bool sparse_tile_ok(uint32_t n_tile);
cudaError_t sparse_make_tmap(CUtensorMap* out, const int8_t* table, uint32_t CB, uint32_t CT, uint32_t N, uint32_t n_tile,
                             const char** why);
// ... and straight from the canonical table (16-byte aligned), in 64- and 128-wide tiles without a split
float sparse_canonical_plan(uint32_t M, uint32_t CB, uint32_t CT, uint32_t N, int sm_count, uint32_t* n_tile);
cudaError_t sparse_make_canonical_tmap(CUtensorMap* out, const int8_t* lut, uint32_t CB, uint32_t CT, uint32_t N, uint32_t n_tile, const char** why);
cudaError_t sparse_make_idx_tmap(CUtensorMap* out, const uint8_t* idx, uint32_t M, uint32_t CB, uint32_t CT, const char** why);
cudaError_t launch_sparse(const LutArgs& a, const CUtensorMap& lut_map, const CUtensorMap& idx_map, const CUtensorMap& out_map, uint32_t n_tile,
                          uint32_t split, void* partial, uint32_t* counters /* zero between launches */, uint32_t max_ctas,
                          bool fresh_table /* written by a kernel the stream may still run */, bool canonical /* lut_map: sparse_make_canonical_tmap */, uint32_t* dev_err, cudaStream_t s, const char** why);

// A few tokens: the used rows of the canonical table alone (16-byte aligned), row-major fp32 output.
cudaError_t launch_rows(const LutArgs& a, const int8_t* lut, int sm_count, cudaStream_t s);
// ... and the search, in one launch, where rows_search_ok()
bool rows_search_ok(uint32_t M, uint32_t CB, uint32_t CT, uint32_t v, uint32_t N, const float* x);
cudaError_t launch_rows_search(const LutArgs& a, const int8_t* lut, const float* x, const float* centroid, uint32_t v, int sm_count, cudaStream_t s);
float rows_us(uint32_t M, uint32_t CB, uint32_t CT, uint32_t N, int sm_count);

// LUT [CB*CT][N] -> [N][CB*CT]
cudaError_t launch_transpose_lut(const int8_t* lut, int8_t* lut_t, uint32_t rows, uint32_t cols, cudaStream_t s);

// ---- load time: int8 table from centroids x dense weight -------------------------------
struct LutBuildArgs {
    const float* centroid;  // [CB][CT][v]
    const float* weight;    // [K = CB*v][N], row-major
    int8_t* lut;            // out: [CB][CT][N]
    uint32_t* words;        // device scratch: maximum and block counter, zero between calls
    float* scalars;         // mapped host memory: scale, LUT bias
    uint32_t CB, CT, v, N;
};
// Two launches on `s`: abs-max pass, quantising pass.
cudaError_t launch_lut_build(const LutBuildArgs& a, cudaStream_t s, const char** why);

// LUT in the reference's DPU layout (re-tiled along the output features, tile width T) -> canonical.
cudaError_t launch_lut_untile(const int8_t* dpu, int8_t* canonical, uint32_t rows, uint32_t N, uint32_t T,
                              cudaStream_t s, const char** why);

// ---- measurement aid: the int8 tensor rate itself --------------------------------------
// `slabs` x four 128 x n_tile x 32 instructions per CTA, `grid` CTAs; the cycles CTA 0 took land in *d_cycles.
cudaError_t launch_int8_peak(uint32_t n_tile, uint32_t slabs, uint32_t grid, unsigned long long* d_cycles, uint32_t* dev_err,
                             cudaStream_t s, const char** why);

// Activations for timing: token m's sub-vector of codebook cb lies near one of that codebook's centroids, spread evenly over them.
cudaError_t launch_spread_input(const float* centroid, float* x, uint32_t M, uint32_t CB, uint32_t CT, uint32_t v, cudaStream_t s);

// Self-test: a bounded wait on a barrier nobody arrives at; the kernel reports through *dev_err and returns.
cudaError_t launch_stalled_wait(uint32_t polls, uint32_t* dev_err, cudaStream_t s);

// The opt-in to more than 48 KB of dynamic shared memory, asked for once per kernel, device and size (the call takes a
// good part of a microsecond): remembers, per kernel, the largest size asked for on each device.
struct SmemOptIn {
    std::atomic<int> granted[64] = {};
};
template <typename K>
cudaError_t allow_smem(SmemOptIn& memo, K kernel, int bytes) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 64 && memo.granted[dev].load(std::memory_order_relaxed) >= bytes) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess && dev < 64) memo.granted[dev].store(bytes, std::memory_order_relaxed);
    return e;
}

// Driver entry point for tensor-map encoding, resolved through the runtime so the library
// carries no link-time dependency on the driver and loads on machines without one.
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn get_encode_tiled();

// Ordinal of the device whose (or managed) memory this is, -1 for host memory and for what CUDA does not know.
int pointer_device(const void* p);

}  // namespace lutamm
