// lutamm_amm_static_scratch(): the AMM for callers that must not allocate device memory.
//
// Who that is.  Some hosts hand this library a GPU whose memory they have already carved
// up: an inference server that sizes its arenas at start-up and treats any later
// cudaMalloc as a bug (it synchronises the whole device and can fail once memory is
// fragmented), a latency-critical loop that may not block on the allocator, or an embedding
// application that gives a plug-in a fixed set of buffers and nothing else.  The regular
// entry points keep a grow-only scratch arena per context, so their first call at a new
// size allocates.  This one never does: not cudaMalloc/cudaFree, not a pooled or library
// allocator.
//
// How.  The only intermediate of the operator is the closest-centroid index buffer,
// uint8 [n_tokens][num_codebook], written by the search kernel and read by the
// gather-accumulate kernel.  Here it lives in a file-scope __device__ array of fixed size.  The
// kernels' error word is host memory, a static page that the first call on any device maps into
// the devices: a call then clears and reads it without a copy (the memset, the copy back to
// pageable memory and their gaps were 30 us of a 170 us call).  Every GPU that loads this library therefore holds
// LUTAMM_STATIC_SCRATCH_BYTES + 256 bytes of device memory from module load until the
// process exits, whether or not the entry point is ever called.
//
// Rules that follow from one shared array:
//   * n_tokens * num_codebook must not exceed LUTAMM_STATIC_SCRATCH_BYTES; larger problems
//     are rejected with LUTAMM_EINVAL (split the batch);
//   * the array keeps whatever the previous call left in it; the error word is cleared at the
//     start of every call, and the index region is fully rewritten by the search kernel before
//     it is read;
//   * two calls that overlap on the GPU (different streams, different threads, different
//     contexts of one process on one device) race on the array.  Serialise them.
//
// Set-up.  A __device__ array's name is only a host-side handle; the device address comes
// from cudaGetSymbolAddress, per device, with that device current.  The first call on a
// device does this (and maps the error words and sets the kernels' shared-memory attribute); make that first call
// before any stream capture begins, because these set-up calls are not stream operations.
//
// No counterpart in the reference, whose amm_host() allocates (and leaks) its index buffer
// on every call (inference-engine/src/host/amm_host.cpp:19).
#include <atomic>
#include <mutex>
#include <string>

#include "../../include/lutamm.h"
#include "kernels.h"

namespace {

constexpr size_t kHeaderBytes = 256;  // error word, padded so the index region stays 256-byte aligned
static __device__ __align__(256) unsigned char g_static_scratch[kHeaderBytes + LUTAMM_STATIC_SCRATCH_BYTES];

constexpr int kMaxDevices = 64;
std::mutex g_mu;
unsigned char* g_scratch_ptr[kMaxDevices] = {};  // device address of g_static_scratch, per device
// Error words, one per device, 64 bytes apart, and their addresses as the devices see them.
alignas(4096) volatile uint32_t g_err_words[kMaxDevices * 16];
uint32_t* g_err_ptr[kMaxDevices] = {};
bool g_err_mapped = false;
thread_local std::string g_err;

int fail(int code, const std::string& msg) {
    g_err = msg;
    return code;
}

uint32_t sm_count_of(int device) {
    static std::atomic<uint32_t> known[kMaxDevices] = {};
    uint32_t n = known[device].load(std::memory_order_relaxed);
    if (!n) {
        int v = 0;
        n = cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, device) == cudaSuccess && v > 0 ? (uint32_t)v : 148u;
        known[device].store(n, std::memory_order_relaxed);
    }
    return n;
}

// By estimated time: the table's used rows, for few tokens; the tcgen05 kernel on the table as it is; or the CUDA-core
// gather, its narrow tiles of few tokens where wide ones would leave SMs without a CTA.  Laying the table out first, as a
// context does once per layer, was slower at all of 70 sizes (512 tokens 768 -> 3072: 54 us a call against 25; 8192 tokens
// 1024 -> 4096: 116 against 92), and is left for tables that are not 16-byte aligned, which the copy engine cannot read:
// `columns` at a time in what the indices leave of the array.  Over those sizes (1 to 8192 tokens) the choice takes 0.7 %
// more than the fastest form of each, on average.
struct TablePlan {
    bool rows;
    uint32_t direct, columns, gather_cfg;   // direct: tile width
};
TablePlan plan_table(uint32_t M, uint32_t CB, uint32_t CT, uint32_t N, bool aligned, uint32_t sms) {
    const uint32_t cfg = (uint64_t)((M + 63) / 64) * ((N + 255) / 256) < sms ? 4 : 0;
    const float gather = 2.5f + lutamm::gather_us(M, CB, CT, N, cfg, (int)sms), rows = aligned ? lutamm::rows_us(M, CB, CT, N, (int)sms) : 3e38f;
    float table = 3e38f;
    uint32_t columns = 0, direct = 0;
    if (lutamm::umma_supported(CB, CT, N)) {
        if (aligned) {
            table = 6.5f + lutamm::sparse_canonical_plan(M, CB, CT, N, (int)sms, &direct);
        } else {
            const size_t per_column = lutamm::sparse_table_bytes(CB, CT, 1), used = (((size_t)M * CB + 255) / 256) * 256;
            const size_t fit = used < LUTAMM_STATIC_SCRATCH_BYTES ? (LUTAMM_STATIC_SCRATCH_BYTES - used) / per_column : 0;
            columns = fit < N ? (uint32_t)(fit / 64 * 64) : N;
            if (columns) {
                const uint32_t chunks = (N + columns - 1) / columns;
                columns = ((N + chunks - 1) / chunks + 63) / 64 * 64;   // near-equal chunks
                if (columns > N) columns = N;
                uint32_t n_tile, split;
                // a piece: two launches, the layout at 2.5 TB/s, the contraction (measured 768 -> 768 to 512 -> 8192, 1 to 5 pieces)
                const float contraction = lutamm::sparse_default_plan(M, CB, CT, columns, (int)sms, &n_tile, &split, 0, 1);
                table = 3.1f + chunks * (3.7f + (float)per_column * columns / 2.5e6f + contraction);
            }
        }
    }
    const bool contract = table < gather;
    return {rows < table && rows < gather, contract ? direct : 0u, contract ? columns : 0u, cfg};
}

}  // namespace

extern "C" const char* lutamm_static_scratch_last_error(void) { return g_err.c_str(); }

extern "C" int lutamm_amm_static_scratch(int device, void* cuda_stream, const float* input, const float* centroid,
                                         const int8_t* lut, const float* bias, float* output,
                                         const lutamm_index_params* ip, const lutamm_lut_params* lp) {
    using namespace lutamm;
    if (!input || !centroid || !lut || !bias || !output || !ip || !lp) return fail(LUTAMM_EINVAL, "null argument");
    if (device < 0 || device >= kMaxDevices) return fail(LUTAMM_EINVAL, "device ordinal out of range");
    const uint32_t M = ip->n, K = ip->input_feature_len, CB = ip->num_codebook, CT = ip->num_centroid;
    const uint32_t N = lp->output_feature_len;
    if (!K || !CB || !CT || !N || K % CB) return fail(LUTAMM_EINVAL, "bad shape: need input_feature_len % num_codebook == 0 and positive sizes");
    if (ip->sub_vec_len && ip->sub_vec_len != K / CB)
        return fail(LUTAMM_EINVAL, "sub_vec_len != input_feature_len / num_codebook");
    if (lp->num_codebook != CB || lp->num_centroid != CT || lp->n != M)
        return fail(LUTAMM_EINVAL, "index and LUT parameter blocks disagree");
    if (CT > 256) return fail(LUTAMM_EINVAL, "num_centroid > 256 does not fit the uint8 index");
    if (N % 16) return fail(LUTAMM_EINVAL, "output_feature_len must be a multiple of 16");
    if (M == 0) return LUTAMM_OK;
    if ((uint64_t)M * CB > (uint64_t)LUTAMM_STATIC_SCRATCH_BYTES)
        return fail(LUTAMM_EINVAL, "n * num_codebook = " + std::to_string((uint64_t)M * CB) +
                                       " index bytes exceed the static scratch of " +
                                       std::to_string((uint64_t)LUTAMM_STATIC_SCRATCH_BYTES) +
                                       " bytes; split the batch or use lutamm_amm()");

    int prev = -1;
    if (cudaGetDevice(&prev) != cudaSuccess || cudaSetDevice(device) != cudaSuccess)
        return fail(LUTAMM_ECUDA, std::string("cannot select device: ") + cudaGetErrorString(cudaGetLastError()));
    struct Restore {
        int d;
        ~Restore() { if (d >= 0) cudaSetDevice(d); }
    } restore{prev};

    for (const void* p : {(const void*)input, (const void*)centroid, (const void*)lut, (const void*)bias, (const void*)output})
        if (lutamm::pointer_device(p) != device)
            return fail(LUTAMM_EINVAL, "every buffer must be device memory of the selected GPU: this entry point stages nothing");
    if ((reinterpret_cast<uintptr_t>(output) & 15u) || (reinterpret_cast<uintptr_t>(input) & 3u))
        return fail(LUTAMM_EINVAL, "output must be 16-byte aligned, input 4-byte aligned");

    unsigned char* scratch;
    {
        // once per device, with that device current: the symbol's device address
        std::lock_guard<std::mutex> lk(g_mu);
        if (!g_scratch_ptr[device]) {
            void* p = nullptr;
            const cudaError_t e = cudaGetSymbolAddress(&p, g_static_scratch);
            if (e != cudaSuccess || !p)
                return fail(LUTAMM_ECUDA, std::string("cudaGetSymbolAddress(static scratch): ") + cudaGetErrorString(e));
            void* words = const_cast<uint32_t*>(g_err_words);
            if (!g_err_mapped) {
                const cudaError_t re = cudaHostRegister(words, sizeof g_err_words, cudaHostRegisterMapped | cudaHostRegisterPortable);
                if (re != cudaSuccess) return fail(LUTAMM_ECUDA, std::string("cudaHostRegister(error words): ") + cudaGetErrorString(re));
                g_err_mapped = true;
            }
            void* dp = nullptr;
            const cudaError_t pe = cudaHostGetDevicePointer(&dp, words, 0);
            if (pe != cudaSuccess) return fail(LUTAMM_ECUDA, std::string("cudaHostGetDevicePointer: ") + cudaGetErrorString(pe));
            g_err_ptr[device] = static_cast<uint32_t*>(dp) + 16 * device;
            g_scratch_ptr[device] = static_cast<unsigned char*>(p);
        }
        scratch = g_scratch_ptr[device];
    }
    uint32_t* d_err = g_err_ptr[device];
    volatile uint32_t& err_word = g_err_words[16 * device];
    uint8_t* d_idx = scratch + kHeaderBytes;
    cudaStream_t s = static_cast<cudaStream_t>(cuda_stream);

    err_word = 0;
    const char* why = nullptr;
    CcsArgs ca{};
    ca.x = input; ca.centroid = centroid; ca.idx_out = d_idx;
    ca.M = M; ca.K = K; ca.v = K / CB; ca.CB = CB; ca.CT = CT;
    ca.format = LUTAMM_INDEX_U8_ROWMAJOR;
    ca.dev_err = d_err;
    cudaError_t e = launch_ccs(ca, s, &why);
    if (e != cudaSuccess) return fail(LUTAMM_ECUDA, why ? why : (std::string("search launch: ") + cudaGetErrorString(e)));

    LutArgs la{};
    la.idx = d_idx; la.bias = bias; la.out = output; la.acc_out = nullptr;
    la.M = M; la.CB = CB; la.CT = CT; la.N = N;
    la.scale = lp->scale; la.lut_bias = lp->bias;
    const uint32_t sms = sm_count_of(device);
    const TablePlan plan = plan_table(M, CB, CT, N, !(reinterpret_cast<uintptr_t>(lut) & 15u), sms);
    if (plan.rows) {
        e = launch_rows(la, lut, (int)sms, s);
        if (e != cudaSuccess) return fail(LUTAMM_ECUDA, std::string("row gather launch: ") + cudaGetErrorString(e));
    } else if (plan.direct) {
        CUtensorMap idx_map, table_map, out_map;
        e = sparse_make_idx_tmap(&idx_map, d_idx, M, CB, CT, &why);
        if (e == cudaSuccess) e = sparse_make_canonical_tmap(&table_map, lut, CB, CT, N, plan.direct, &why);
        if (e == cudaSuccess) e = make_out_tmap(&out_map, output, M, N, &why);
        // (the table may be what the caller's last kernel writes: its copies wait for the search, and that for the caller)
        if (e == cudaSuccess) e = launch_sparse(la, table_map, idx_map, out_map, plan.direct, 1, nullptr, nullptr, sms, true, true, d_err, s, &why);
        if (e != cudaSuccess) return fail(LUTAMM_ECUDA, why ? why : (std::string("tcgen05 launch: ") + cudaGetErrorString(e)));
    } else if (plan.columns) {
        // the tcgen05 kernel on as many columns at a time as the rest of the array holds of its layout of the table
        int8_t* table = reinterpret_cast<int8_t*>(d_idx + (((size_t)M * CB + 255) / 256) * 256);
        CUtensorMap idx_map;
        e = sparse_make_idx_tmap(&idx_map, d_idx, M, CB, CT, &why);
        for (uint32_t n0 = 0; n0 < N && e == cudaSuccess; n0 += plan.columns) {
            la.N = N - n0 < plan.columns ? N - n0 : plan.columns;
            la.bias = bias + n0;
            la.out = output + n0;
            const uint32_t left = N - n0 - la.N;
            la.next_ctas = left ? sparse_table_ctas(CB, CT, left < plan.columns ? left : plan.columns) : 0;   // the next piece's layout
            la.next_per_sm = 8;
            uint32_t n_tile, split;
            sparse_default_plan(M, CB, CT, la.N, (int)sms, &n_tile, &split, 0, 1);
            CUtensorMap table_map, out_map;
            // (the second table and on: the contraction in front began when all that the caller had queued was complete)
            e = launch_sparse_table(lut, table, CB, CT, la.N, n0, N, n0 > 0, s);
            if (e == cudaSuccess) e = sparse_make_tmap(&table_map, table, CB, CT, la.N, n_tile, &why);
            if (e == cudaSuccess) e = make_out_tmap(&out_map, la.out, M, la.N, &why, N);
            if (e == cudaSuccess) e = launch_sparse(la, table_map, idx_map, out_map, n_tile, 1, nullptr, nullptr, sms, true, false, d_err, s, &why);
        }
        if (e != cudaSuccess) return fail(LUTAMM_ECUDA, why ? why : (std::string("tcgen05 launch: ") + cudaGetErrorString(e)));
    } else {
        // The gather-accumulate kernel reads the LUT in its canonical layout through a tensor map encoded on the host (no
        // device memory involved).
        const uint32_t cfg = plan.gather_cfg;
        CUtensorMap map;
        e = gather_make_tmap(&map, lut, CB, CT, N, cfg, &why);
        if (e != cudaSuccess) return fail(LUTAMM_ECUDA, why ? why : cudaGetErrorString(e));
        e = launch_gather(la, map, cfg, d_err, s, &why);
        if (e != cudaSuccess) return fail(LUTAMM_ECUDA, why ? why : (std::string("gather launch: ") + cudaGetErrorString(e)));
    }

    e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return fail(LUTAMM_ECUDA, std::string("cudaStreamSynchronize: ") + cudaGetErrorString(e));
    if (err_word) return fail(LUTAMM_EDEVICE, "a kernel gave up on a bounded wait; output is not valid");
    return LUTAMM_OK;
}
