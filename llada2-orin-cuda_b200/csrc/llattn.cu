// C ABI of libllattn.so (see include/llattn.h): argument checking, the host-side work planner and the kernel
// launches. No torch types, no exit(): every failure comes back as a status code plus a thread-local message.
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <algorithm>
#include <atomic>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <cstdlib>
#include <cmath>
#include <cstdint>
#include <mutex>
#include <new>
#include <vector>

#include "llattn.h"
#include "common.cuh"
#include "kv_commit.cuh"
#include "attn_kernel.cuh"
#include "merge_kernel.cuh"
#include "qkv_prepare.cuh"
#include "dense_i8.cuh"

namespace {

thread_local char g_err[512] = "";

int fail(int code, const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
    return code;
}

#define CU(call)                                                                                  \
    do {                                                                                          \
        cudaError_t e_ = (call);                                                                  \
        if (e_ != cudaSuccess) return fail(LLATTN_ECUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
    } while (0)

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
inline cudaStream_t as_stream(void* s) { return static_cast<cudaStream_t>(s); }

}  // namespace

// ====================================================================================================== context

struct llattn_ctx {
    int device = 0;
    int num_sms = 0;
    int* err_word = nullptr;          // device
    void* workspace = nullptr;        // device: partial results (grow-only)
    size_t workspace_bytes = 0;
    void* stage = nullptr;            // device staging for the host-buffer entry point: two slots (grow-only)
    size_t stage_bytes = 0, stage_slot_bytes = 0;
    bool host_ready = false;          // copy streams and events of the host-buffer path exist
    int host_slot = 0;
    cudaStream_t s_in = nullptr, s_out = nullptr;
    cudaEvent_t ev_in[2] = {}, ev_comp[2] = {}, ev_out[2] = {};
    std::mutex mu;
};

struct llattn_plan {
    llattn_ctx* ctx = nullptr;
    llattn_plan_stats stats{};
    void* dev_blob = nullptr;         // run descriptors, per-CTA ranges, each CTA's first run (fixed section offsets)
    void* host_blob = nullptr;        // pinned mirror: llattn_plan_update fills it and copies it up asynchronously
    size_t blob_bytes = 0, off_items = 0, off_cta = 0, off_first = 0;
    size_t cap_seqs = 0, cap_items = 0, cap_tiles = 0;
    int launch_ctas = 0;              // grid of every launch of this plan (CTAs beyond the used ones find no items)
    int ntiles = 0;                   // output tiles of the plan as it is now
    cudaEvent_t ev_upload = nullptr;
    bool upload_pending = false;
    const llattn::RunDesc* d_items = nullptr;
    const int32_t* d_cta_first = nullptr;
    const llattn::RunDesc* d_first = nullptr;
};

namespace {

struct DeviceGuard {
    int prev = -1;
    bool ok = true;
    explicit DeviceGuard(int dev) {
        if (cudaGetDevice(&prev) != cudaSuccess) { ok = false; return; }
        if (prev != dev && cudaSetDevice(dev) != cudaSuccess) ok = false;
    }
    ~DeviceGuard() { if (prev >= 0) cudaSetDevice(prev); }
};

// A launch that may start before the kernel ahead of it in the stream has run out; its kernel waits with griddepcontrol.wait before it reads
// or writes anything. Behind a kernel that does not allow it earlier, it takes its place when the last CTA of that one has left, and the
// launch's own latency is hidden: every kernel of this library but the cooperative attention goes this way. In a graph, the same build without
// and with the attribute: commit of 64 blocks 4.05 / 3.9 us, 32 tokens through the projection 3.7 / 3.5, operator pair at 2 K tokens 14.1 / 13.7,
// a 20-layer step of one sequence at 8 K tokens 441.4 / 439.3. Calls one after the other through the Python binding, whose host time of 5 to
// 7 us covers the two short ones: pair 16.1 / 14.5, 2048 tokens through the projection 33.0 / 31.0, a first pass over four prompts of 13 blocks 29.3 / 27.1.
// Under capture the edge in front of the kernel becomes a programmatic one.
template <typename... KArgs>
cudaError_t launch_dependent_smem(void (*kernel)(KArgs...), dim3 grid, int threads, int smem, cudaStream_t stream, KArgs... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid; cfg.blockDim = dim3(threads); cfg.stream = stream; cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
    if (e != cudaSuccess) cudaGetLastError();  // reported here, not to whoever asks next
    return e;
}
template <typename... KArgs>
cudaError_t launch_dependent(void (*kernel)(KArgs...), dim3 grid, int threads, cudaStream_t stream, KArgs... args) {
    return launch_dependent_smem(kernel, grid, threads, 0, stream, args...);
}

int ensure_kernel_attrs() {
    static std::mutex mu;
    static bool done[64] = {};
    int dev = 0;
    CU(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(mu);
    if (dev < 64 && done[dev]) return LLATTN_OK;
    CU(cudaFuncSetAttribute(llattn::attn_tile_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, llattn::ATTN_SMEM_BYTES));
    CU(cudaFuncSetAttribute(llattn::attn_tile_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, llattn::ATTN_SMEM_BYTES));
    CU(cudaFuncSetAttribute(llattn::attn_tile_kernel<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, llattn::ATTN_SMEM_BYTES));
    if (dev < 64) done[dev] = true;
    return LLATTN_OK;
}

int grow(void** p, size_t* have, size_t need) {
    if (need <= *have) return LLATTN_OK;
    if (*p) { CU(cudaFree(*p)); *p = nullptr; *have = 0; }
    const size_t want = need + need / 4;
    if (cudaMalloc(p, want) != cudaSuccess) {
        cudaGetLastError();
        return fail(LLATTN_ENOMEM, "cudaMalloc of %zu bytes failed", want);
    }
    *have = want;
    return LLATTN_OK;
}

}  // namespace

extern "C" {

const char* llattn_version(void) { return "llattn 0.1 (sm_100a)"; }
const char* llattn_last_error(void) { return g_err; }

int llattn_pick_bpc(int nblocks, int nbatch) {
    if (nbatch < 1) nbatch = 1;
    const int want = nbatch >= 4 ? 1 : 4 / nbatch;
    return std::max(1, (nblocks + want - 1) / want);
}
int llattn_chunks_for(int nblocks, int bpc) { return nblocks <= 0 ? 1 : (nblocks + bpc - 1) / bpc; }
int llattn_tile_units(void) { return llattn::TILE_UNITS; }

// ------------------------------------------------------------------------------------------------------ commit

namespace {
// Few blocks: 512 threads a record, for the shortest chain. They fit on an SM three at a time (40 registers), CTAs of 256 threads
// four at a time (56), so records pass faster through the latter once there are many waves of them: from two waves of the
// 256-thread form on, twice as many blocks as there are SMs (a block is four CTAs). 512 / 256 threads in a graph: 1 block 3.1 /
// 3.8 us, 64 4.4 / 4.6, 111 and 112 (the second wave of 512) 5.7 and 6.7 / 5.7 and 6.8, 128 6.9 / 7.0, 149 7.9 / 8.2, 222 9.4 / 9.6,
// 296 11.8 / 12.0, 384 15.3 / 14.9, 1024 37.5 / 34.8, 2048 74.7 / 67.9.
int launch_commit(const void* Kf, const void* Vf, void* records, const int32_t* pages, int max_blocks, int blk, int nb, void* stream) {
    int dev = 0, sms = 0;
    CU(cudaGetDevice(&dev));
    CU(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const dim3 grid(llattn::NKV, nb);
    const half *k = static_cast<const half*>(Kf), *v = static_cast<const half*>(Vf);
    uint8_t* r = static_cast<uint8_t*>(records);
    if (nb <= 2 * sms) CU(launch_dependent(llattn::kv_commit_kernel<512>, grid, 512, as_stream(stream), k, v, r, pages, max_blocks, blk));
    else CU(launch_dependent(llattn::kv_commit_kernel<256>, grid, 256, as_stream(stream), k, v, r, pages, max_blocks, blk));
    return LLATTN_OK;
}
}  // namespace

int llattn_kv_commit(const void* Kf, const void* Vf, void* cache, int max_blocks, int blk, int nb, void* stream) {
    if (!Kf || !Vf || !cache) return fail(LLATTN_EINVAL, "kv_commit: null pointer");
    if (nb < 0 || blk < 0 || max_blocks <= 0 || blk + nb > max_blocks)
        return fail(LLATTN_EINVAL, "kv_commit: blocks [%d, %d) outside a cache of %d blocks", blk, blk + nb, max_blocks);
    if (!aligned16(Kf) || !aligned16(Vf) || !aligned16(cache)) return fail(LLATTN_EINVAL, "kv_commit: pointers must be 16-byte aligned");
    if (nb == 0) return LLATTN_OK;
    if (nb > 65535) return fail(LLATTN_EINVAL, "kv_commit: at most 65535 blocks per call");
    return launch_commit(Kf, Vf, cache, nullptr, max_blocks, blk, nb, stream);
}

int llattn_kv_commit_paged(const void* Kf, const void* Vf, void* pool, const int32_t* pages, int nb, void* stream) {
    if (!Kf || !Vf || !pool || !pages) return fail(LLATTN_EINVAL, "kv_commit_paged: null pointer");
    if (nb < 0 || nb > 65535) return fail(LLATTN_EINVAL, "kv_commit_paged: nb must be in [0, 65535]");
    if (!aligned16(Kf) || !aligned16(Vf) || !aligned16(pool)) return fail(LLATTN_EINVAL, "kv_commit_paged: pointers must be 16-byte aligned");
    if (nb == 0) return LLATTN_OK;
    return launch_commit(Kf, Vf, pool, pages, 0, 0, nb, stream);
}

// ------------------------------------------------------------------------------------------------------ producer

namespace {
int launch_prepare(const float* qkv, const int32_t* pos, const float* gq, const float* gk, float eps, const float* inv_freq,
                   void* q, void* k, void* v, int T, void* records, const int32_t* pages, int max_blocks, int blk, void* stream) {
    llattn::PrepArgs a{qkv, pos, gq, gk, inv_freq, eps, static_cast<half*>(q), static_cast<half*>(k), static_cast<half*>(v), T,
                       static_cast<uint8_t*>(records), pages, max_blocks, blk};
    const int blocks = (T + llattn::BLK - 1) / llattn::BLK;
    using namespace llattn;
    int dev = 0, sms = 0;
    if (records) { CU(cudaGetDevice(&dev)); CU(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)); }
    if (!records) CU(launch_dependent(qkv_prepare_kernel<false, PREP_THREADS>, dim3(blocks, 6 * prep_parts(PREP_THREADS)), PREP_THREADS, as_stream(stream), a));
    else if (9 * (long long)blocks <= 4 * sms)
        CU(launch_dependent(qkv_prepare_kernel<true, PREP_FEW_THREADS>, dim3(blocks, NKV + 4 * prep_parts(PREP_FEW_THREADS)), PREP_FEW_THREADS, as_stream(stream), a));
    else CU(launch_dependent(qkv_prepare_kernel<true, PREP_THREADS>, dim3(blocks, NKV + 4 * prep_parts(PREP_THREADS)), PREP_THREADS, as_stream(stream), a));
    return LLATTN_OK;
}
}  // namespace

int llattn_qk_norm_rope(const float* qkv, const int32_t* pos, const float* gq, const float* gk, float eps,
                        const float* inv_freq, void* q, void* k, void* v, int T, void* stream) {
    if (!qkv || !pos || !gq || !gk || !inv_freq || !q || !k || !v) return fail(LLATTN_EINVAL, "qk_norm_rope: null pointer");
    if (T < 0 || T > 1 << 24) return fail(LLATTN_EINVAL, "qk_norm_rope: T = %d", T);
    if (!aligned16(k) || !aligned16(v)) return fail(LLATTN_EINVAL, "qk_norm_rope: k and v must be 16-byte aligned");
    if (T == 0) return LLATTN_OK;
    return launch_prepare(qkv, pos, gq, gk, eps, inv_freq, q, k, v, T, nullptr, nullptr, 0, 0, stream);
}

int llattn_qkv_prepare_commit(const float* qkv, const int32_t* pos, const float* gq, const float* gk, float eps,
                              const float* inv_freq, void* q, void* k, void* v, int nb, void* cache, const int32_t* pages,
                              int max_blocks, int blk, void* stream) {
    if (!qkv || !pos || !gq || !gk || !inv_freq || !q || !k || !v || !cache) return fail(LLATTN_EINVAL, "qkv_prepare_commit: null pointer");
    if (nb < 0 || nb > 65535) return fail(LLATTN_EINVAL, "qkv_prepare_commit: nb must be in [0, 65535]");
    if (!pages && (blk < 0 || max_blocks <= 0 || blk + nb > max_blocks))
        return fail(LLATTN_EINVAL, "qkv_prepare_commit: blocks [%d, %d) outside a cache of %d blocks", blk, blk + nb, max_blocks);
    if (!aligned16(k) || !aligned16(v) || !aligned16(cache)) return fail(LLATTN_EINVAL, "qkv_prepare_commit: k, v and cache must be 16-byte aligned");
    if (nb == 0) return LLATTN_OK;
    return launch_prepare(qkv, pos, gq, gk, eps, inv_freq, q, k, v, nb * llattn::BLK, cache, pages, max_blocks, blk, stream);
}

// ------------------------------------------------------------------------------------------------------ consumer
// The attention-output projection on the int8 activations the merge kernel writes.

namespace {
// Up to this many tokens the strip kernel may be the faster one: it reads the weights once per 32 tokens, with every SM.
constexpr int DENSE_STRIP_MAX_TOKENS = 64;

// Strip kernel or 16-token tiles. One strip CTA fills an SM (512 threads of 128 registers), so its time goes with the rows too:
// 2048 rows of K = 2048 are one wave (3.2 us for 16 tokens, 8.0 as tiles), 4096 two (5.3 and 8.3), 16,384 seven (17.5 and 9.7; 64
// tokens at K = 512 26.0, in 64-token tiles 7.2). Both as measured in a graph over 2048 .. 32,768 rows, K = 256 .. 8192 and 1 .. 64
// tokens, in hundredths of a microsecond: a wave of strips per sixteen groups and the tokens in it (a partly filled last wave
// counts half), and the serial groups of a tile. The choice is within 11 % of the faster one everywhere there. (Rows and tokens
// beyond one wave of 16-token tiles need no case of their own: the strips have lost long before.)
bool dense_strips_win(int rows, int K, int ntokens, int sms) {
    const int batches = (ntokens + llattn::DS_TOK - 1) / llattn::DS_TOK, per_cta = (ntokens + batches - 1) / batches;
    const double groups = K / llattn::DN_GROUP, live = std::min(groups, double(llattn::DS_WARPS));          // live: warps with a group
    const double ctas = double(rows / 16) * batches, waves = std::max(1.0, (ctas / sms + std::ceil(ctas / sms)) / 2);
    const double wave = 110 + 2 * live + per_cta * (0.9 + 0.14 * live);
    return 130 + waves * std::max(1.0, groups / llattn::DS_WARPS) * wave <= 210 + 37 * groups;
}

// Tokens per CTA of the tcgen05 form, or 0 where the mma.sync tiles are the faster ones. A CTA of the former fills an SM and has a
// long start (tensor memory, four roles, sixteen groups' factors), so it wins with the groups and with the tokens; the line follows
// both sides' measured costs in microseconds, in a graph over 1024 .. 4096 rows, K = 256 .. 4096 and 96 .. 4096 tokens. A CTA walks its
// tiles without ending, so that a further one costs less than the first. 2048 rows, tiles / tcgen05 with 32, 64 and 128 tokens a CTA:
//   K = 2048   160 tokens 11.2 / 11.0, 12.3, 16.9    320  16.7 / 18.1, 12.2, 16.9    640 26.6 / 25.2, 21.4, 17.0   2048 49.7 / -, 39.1, 31.7
//   K = 512    320 tokens  6.6 / 9.2, 7.1, 9.3      2048  18.2 / -, 19.2, 15.5
// Over those 198 sizes the choice costs 0.6 % over the fastest form in the mean (10 % at most, where the tiles' cost is off) and a call
// that takes the tcgen05 form is at most 1 % slower than its tiles.
int dense_wide_tokens(int rows, int K, int ntokens, int sms) {
    if (ntokens <= 32) return 0;
    const double groups = K / llattn::DN_GROUP, row_tiles = rows / llattn::DN_ROWS;
    auto ctas = [&](int tok) { return row_tiles * ((ntokens + tok - 1) / tok); };
    double best;
    if (ctas(16) <= sms) best = 2.1 + 0.38 * groups;
    else if (ctas(32) <= sms) best = 2.3 + 0.54 * groups;
    else if (ctas(64) <= sms) best = 2.6 + 0.88 * groups;
    else {                                     // two CTAs an SM. A partly filled last wave counts half; behind six others, which have
                                               // drifted apart by then, a fifth (K = 768, 16,384 rows, 1184 tokens: 87.3 measured, 98 by a half, 96 by a fifth)
        const double waves = ctas(64) / (2 * sms), idle = std::ceil(waves) - waves;
        best = std::max(1.0, waves + idle * (waves > 6 ? 0.2 : 0.5)) * (2.9 + 1.42 * groups);
    }
    int wide = 0;
    // Two groups: the tiles. Up to six in many waves stay with them as well, a line drawn for a CTA per tile: since CTAs walk their tiles, 128
    // tokens a CTA are the faster form there too (as tiles / so: 12,288 rows of K = 768, 1800 tokens 97.7 / 86.5 us, 16,384 rows, 1184 tokens
    // 87.3 / 74.6, 8192 rows, 4096 tokens 144 / 111, 16,384 rows of K = 512, 2048 tokens 108.5 / 94.4, of K = 384 94 / 84).
    if (groups <= 2 || (groups <= 6 && ctas(64) > 6 * 2 * sms)) return 0;
    auto consider = [&](int tok, double start, double group, double more, double group_more) {
        const double cost = start + group * groups + (std::ceil(ctas(tok) / sms) - 1) * (more + group_more * groups);
        if (cost < best) { best = cost; wide = tok; }
    };
    consider(32, 4.7, 0.388, 1.4, 0.375);
    consider(64, 5.3, 0.455, 2.2, 0.445);
    consider(128, 6.6, 0.68, 2.6, 0.685);
    return wide;
}

// Which kernel takes a call and the tokens of a CTA, by the sizes and the SM count alone. `tcgen05`: that kernel can be launched.
struct DenseForm {
    int kernel, tokens;
};
DenseForm dense_form(int rows, int K, int ntokens, int sms, bool tcgen05 = true) {
    if (ntokens <= DENSE_STRIP_MAX_TOKENS && dense_strips_win(rows, K, ntokens, sms)) return {LLATTN_DENSE_STRIPS, llattn::DS_TOK};
    if (tcgen05)
        if (const int wide = dense_wide_tokens(rows, K, ntokens, sms)) return {LLATTN_DENSE_TCGEN05, wide};
    // The largest tile is the cheapest per token, as long as the tiles fill the chip: with smaller ones while they do not.
    // 2048 x 2048, in a graph: 65 .. 144 tokens 16.2 .. 16.6 us with 64 tokens a tile, 8.1 .. 8.7 with 16; 160 .. 288 tokens 16.7 and
    // 11.3 .. 11.8 (32); at 512 tokens 16.8 (64) and 17.3 (32), at 1024 26.4 and 30.7.
    // Never a tile larger than the tokens: 32,768 rows of K = 8192 and one token 43 us with 16, 85 with 64.
    const long long row_tiles = rows / llattn::DN_ROWS;
    if (ntokens <= 16 || row_tiles * ((ntokens + 15) / 16) <= sms) return {LLATTN_DENSE_TILES, 16};
    if (ntokens <= 32 || row_tiles * ((ntokens + 31) / 32) <= sms) return {LLATTN_DENSE_TILES, 32};
    return {LLATTN_DENSE_TILES, 64};
}

int check_dense_sizes(int rows, int K, int ntokens) {
    if (ntokens < 0 || ntokens > 1 << 22) return fail(LLATTN_EINVAL, "dense_w4a8: ntokens = %d", ntokens);
    if (rows <= 0 || rows % llattn::DN_ROWS || K <= 0 || K % llattn::DN_GROUP || K > 1 << 20 || rows > 1 << 20)
        return fail(LLATTN_EINVAL, "dense_w4a8: rows = %d, K = %d (both multiples of 128)", rows, K);
    return LLATTN_OK;
}
}  // namespace

int llattn_dense_preview(int rows, int K, int ntokens, int num_sms, int* kernel, int* tokens_per_cta) {
    if (!kernel || !tokens_per_cta) return fail(LLATTN_EINVAL, "dense_preview: null pointer");
    if (int rc = check_dense_sizes(rows, K, ntokens)) return rc;
    if (ntokens < 1 || num_sms < 1) return fail(LLATTN_EINVAL, "dense_preview: ntokens and num_sms must be positive");
    const DenseForm f = dense_form(rows, K, ntokens, num_sms);
    *kernel = f.kernel;
    *tokens_per_cta = f.tokens;
    return LLATTN_OK;
}

int llattn_dense_w4a8(const void* W, const int8_t* q, const float* s, const int32_t* sum, float* Y, int ntokens, int rows, int K,
                      int* err_word, void* stream) {
    if (!W || !q || !s || !sum || !Y) return fail(LLATTN_EINVAL, "dense_w4a8: null pointer");
    if (int rc = check_dense_sizes(rows, K, ntokens)) return rc;
    if (ntokens == 0) return LLATTN_OK;
    if (!aligned16(W) || !aligned16(q)) return fail(LLATTN_EINVAL, "dense_w4a8: W and q must be 16-byte aligned");
    const llattn::DenseParams p{static_cast<const uint8_t*>(W), q, s, sum, Y, ntokens, rows, K, err_word};
    static std::once_flag once[64];
    static std::atomic<int> split_ok[64];      // 1: the tcgen05 kernels have the registers that their roles divide
    int dev = 0;
    CU(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64)
        std::call_once(once[dev], [dev] {
            bool ok = true;
            auto wide = [&](auto* kernel, int smem) {
                cudaFuncAttributes a{};
                ok = ok && cudaFuncGetAttributes(&a, kernel) == cudaSuccess && a.numRegs >= llattn::DW_LAUNCH_REGS;
                cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
            };
            wide(llattn::dense_wide_kernel<32, false>, llattn::DenseWide<32>::SMEM); wide(llattn::dense_wide_kernel<32, true>, llattn::DenseWide<32>::SMEM);
            wide(llattn::dense_wide_kernel<64, false>, llattn::DenseWide<64>::SMEM);
            wide(llattn::dense_wide_kernel<128, false>, llattn::DenseWide<128>::SMEM);
            split_ok[dev] = ok;
            cudaFuncSetAttribute(llattn::dense_strip_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, llattn::DS_SMEM_BYTES);
            cudaFuncSetAttribute(llattn::dense_tile_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, llattn::DenseTile<16>::SMEM);
            cudaFuncSetAttribute(llattn::dense_tile_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, llattn::DenseTile<32>::SMEM);
            cudaFuncSetAttribute(llattn::dense_tile_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, llattn::DenseTile<64>::SMEM);
        });
    int sms = 0;
    CU(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const DenseForm f = dense_form(rows, K, ntokens, sms, dev >= 0 && dev < 64 && split_ok[dev]);
    const bool strips = f.kernel == LLATTN_DENSE_STRIPS;
    const dim3 tiles(rows / (strips ? 16 : llattn::DN_ROWS), (ntokens + f.tokens - 1) / f.tokens);
    // With 32 tokens a CTA and no more tiles than SMs, a CTA per tile in a kernel without the loop over them: 160 tokens 10.0 us, 10.4 with it.
    const bool one = f.tokens == 32 && (long long)tiles.x * tiles.y <= sms;
    const dim3 grid = f.kernel == LLATTN_DENSE_TCGEN05 && !one ? dim3(unsigned(std::min<long long>(sms, (long long)tiles.x * tiles.y))) : tiles;
    cudaError_t e = cudaSuccess;
    auto launch = [&](auto* kernel, int threads, int smem) { e = launch_dependent_smem(kernel, grid, threads, smem, as_stream(stream), p); };
    if (strips) launch(llattn::dense_strip_kernel, llattn::DS_THREADS, llattn::DS_SMEM_BYTES);
    else if (f.kernel == LLATTN_DENSE_TCGEN05) {
        if (f.tokens == 32) launch(one ? llattn::dense_wide_kernel<32, true> : llattn::dense_wide_kernel<32, false>, llattn::DW_THREADS, llattn::DenseWide<32>::SMEM);
        else if (f.tokens == 64) launch(llattn::dense_wide_kernel<64, false>, llattn::DW_THREADS, llattn::DenseWide<64>::SMEM);
        else launch(llattn::dense_wide_kernel<128, false>, llattn::DW_THREADS, llattn::DenseWide<128>::SMEM);
    } else {
        if (f.tokens == 16) launch(llattn::dense_tile_kernel<16>, llattn::DT_THREADS, llattn::DenseTile<16>::SMEM);
        else if (f.tokens == 32) launch(llattn::dense_tile_kernel<32>, llattn::DT_THREADS, llattn::DenseTile<32>::SMEM);
        else launch(llattn::dense_tile_kernel<64>, llattn::DT_THREADS, llattn::DenseTile<64>::SMEM);
    }
    CU(e);
    return LLATTN_OK;
}

int llattn_dense_error_word(int** word) {
    if (!word) return fail(LLATTN_EINVAL, "dense_error_word: null pointer");
    *word = nullptr;
    void* p = nullptr;
    CU(cudaGetSymbolAddress(&p, llattn::g_dense_err));
    *word = static_cast<int*>(p);
    return LLATTN_OK;
}

int llattn_dense_status(void* stream, int* code) {
    if (!code) return fail(LLATTN_EINVAL, "dense_status: null pointer");
    *code = 0;
    CU(cudaStreamSynchronize(as_stream(stream)));
    CU(cudaMemcpyFromSymbol(code, llattn::g_dense_err, sizeof(int)));
    if (*code) {
        const int zero = 0;
        CU(cudaMemcpyToSymbol(llattn::g_dense_err, &zero, sizeof(int)));
        return fail(LLATTN_EDEVICE, "a projection's wait ran out (error bits 0x%x): its Y is incomplete", *code);
    }
    return LLATTN_OK;
}

}  // extern "C"

#include "llattn_attention.inl"
#include "kvpool.inl"

// ====================================================================================================== no-allocation entry point
// Scratch for llattn_attention_static: partial results (un-normalised O, reference maximum, row sum) of up to
// STATIC_MAX_SLOTS runs. It lives in the library image, so every GPU that loads the library holds these bytes until the
// process exits, and every call on a device shares them.
namespace {
constexpr int STATIC_MAX_SLOTS = 160;                                  // 148 SMs worth of runs for one query block, rounded up
constexpr int STATIC_MAX_QBLOCKS = 16;                                 // a prefill pass of the reference engine
constexpr size_t STATIC_SLOT_FLOATS = size_t(llattn::QR) * llattn::D + 2 * llattn::QR;   // 16640 floats = 66560 B
}  // namespace
static __device__ __align__(256) float g_static_scratch[STATIC_MAX_SLOTS * STATIC_SLOT_FLOATS];   // 10.16 MiB

namespace {
struct StaticSetup { float* scratch = nullptr; int num_sms = 0; bool ready = false; };
StaticSetup g_static[64];
std::mutex g_static_mu;

// Once per device, with that device current: resolve the DEVICE address of the scratch array. In host code the
// array's name is only a stand-in symbol; handing it to a kernel would make the kernel dereference a host address.
int static_setup(int dev, StaticSetup** out) {
    if (dev < 0 || dev >= 64) return fail(LLATTN_EINVAL, "attention_static: device index %d not supported", dev);
    std::lock_guard<std::mutex> lk(g_static_mu);
    StaticSetup& st = g_static[dev];
    if (!st.ready) {
        float* ptr = nullptr;
        cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_static_scratch);
        if (e != cudaSuccess || !ptr) return fail(LLATTN_ECUDA, "attention_static: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
        e = cudaDeviceGetAttribute(&st.num_sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return fail(LLATTN_ECUDA, "attention_static: cudaDeviceGetAttribute: %s", cudaGetErrorString(e));
        st.scratch = ptr;
        st.ready = true;
    }
    *out = &st;
    return LLATTN_OK;
}
}  // namespace

extern "C" int llattn_attention_static(const void* Q, const void* Kf, const void* Vf, const void* cache, int max_blocks,
                                       int nblocks, int nb, float scale, void* O16, float* O32, float* LSE, int8_t* q8,
                                       float* s8, int32_t* sum8, int* err_word, void* stream) {
    using namespace llattn;
    if (!Q || !Kf || !Vf) return fail(LLATTN_EINVAL, "attention_static: Q, Kf and Vf are required");
    if (!O16 && !O32 && !LSE && !q8) return fail(LLATTN_EINVAL, "attention_static: no output requested");
    if (q8 && (!s8 || !sum8)) return fail(LLATTN_EINVAL, "attention_static: q8 needs s8 and sum8");
    if (nb < 1 || nb > STATIC_MAX_QBLOCKS)
        return fail(LLATTN_EINVAL, "attention_static: %d query blocks; the built-in scratch serves 1..%d per call", nb, STATIC_MAX_QBLOCKS);
    if (nblocks < 0 || max_blocks < 0 || nblocks + nb - 1 > max_blocks)
        return fail(LLATTN_EINVAL, "attention_static: %d blocks visible, cache holds %d", nblocks + nb - 1, max_blocks);
    if (nblocks + nb - 1 > 0 && !cache) return fail(LLATTN_EINVAL, "attention_static: null cache with committed blocks");
    if (!aligned16(Q) || !aligned16(Kf) || !aligned16(Vf) || !aligned16(cache) || !aligned16(O16) || !aligned16(O32))
        return fail(LLATTN_EINVAL, "attention_static: pointers must be 16-byte aligned");
    int dev = -1;
    CU(cudaGetDevice(&dev));
    StaticSetup* st = nullptr;
    if (int rc = static_setup(dev, &st)) return rc;
    if (int rc = ensure_kernel_attrs()) return rc;
    // split each (query block, kv head) into runs so that about one run lands on every SM, within the scratch's slots
    const int nbl = nblocks + nb - 1;
    const int want = std::max(1, std::min(STATIC_MAX_SLOTS / (NKV * nb), (st->num_sms + NKV * nb - 1) / (NKV * nb)));
    int bpc = std::max(1, (nbl + want - 1) / want);
    bpc = std::max(bpc, std::min(nbl, 8));                       // at least two 128-key tiles per run when there are that many
    bpc = (bpc + TILE_UNITS - 1) / TILE_UNITS * TILE_UNITS;      // cuts on tile boundaries
    const int nchunks = llattn_chunks_for(nbl, bpc);
    if (NKV * nchunks * nb > STATIC_MAX_SLOTS)
        return fail(LLATTN_ENOMEM, "attention_static: %d partial slots needed, the built-in scratch holds %d", NKV * nchunks * nb, STATIC_MAX_SLOTS);
    const size_t ns = size_t(NKV) * nchunks * nb;
    float* Opart = st->scratch;
    float* Mpart = Opart + ns * QR * D;
    float* Lpart = Mpart + ns * QR;
    KParams p{};
    p.Q = static_cast<const half*>(Q); p.Kf = static_cast<const half*>(Kf); p.Vf = static_cast<const half*>(Vf);
    p.Opart = Opart; p.Mpart = Mpart; p.Lpart = Lpart;
    p.sl2 = (scale > 0.f ? scale : 0.08838834764831845f) * 1.4426950408889634f;
    p.err = err_word;
    p.ref_seq = SeqDesc{static_cast<const uint8_t*>(cache), nullptr, max_blocks, nblocks, nb, 0};
    p.ref_bpc = bpc;
    p.ref_nchunks = nchunks;
    CU(launch_dependent_smem(attn_tile_kernel<false>, dim3(NKV * nchunks * nb), ATTN_THREADS, ATTN_SMEM_BYTES, as_stream(stream), p));
    MergeOut o{static_cast<half*>(O16), O32, LSE, q8, s8, sum8};
    CU(launch_dependent(
        nchunks > FOLD_PART ? combine_ref_kernel<true> : combine_ref_kernel<false>, dim3(NKV, QR / MERGE_ROWS, nb), MERGE_THREADS, as_stream(stream),
        static_cast<const float*>(Opart), static_cast<const float*>(Mpart), static_cast<const float*>(Lpart), nchunks, nblocks, bpc, o));
    return LLATTN_OK;
}

// ====================================================================================================== wait self-test
// What a kernel of this library does when a wait can never complete, shown without making any real kernel fail: four
// warps wait on barriers nobody will ever arrive on, a fifth on a counter nobody counts into (the wait a CTA does for
// the other runs of a split tile). Warp 0 has `limit_ns` (a millisecond in the test); when its wait runs out it raises
// the CTA's abort flag, as every role of the attention kernel does, and the other warps - whose own limit is the
// kernels' two seconds - see the flag at their next poll and leave too. Then the fifth warp waits on its counter once
// more, alone and with the short limit, to show that wait running out by itself. Of a sixth warp half of the lanes wait on a barrier
// whose phase is complete and half on one that nobody arrives on: it has to leave its wait with one answer, no, in all lanes.
// Every warp reports through the error word, the kernel returns normally and the context stays usable.
namespace llattn {
__device__ int selftest_counter;       // nothing ever counts in here

__global__ void __launch_bounds__(192) wait_selftest_kernel(unsigned long long limit_ns, int* err, unsigned long long* waited_ns) {
    __shared__ uint64_t bars[5];
    __shared__ int abort_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 5; ++i) ptx::mbar_init(ptx::smem_u32(&bars[i]), 1);
        ptx::fence_mbar_init();
        ptx::mbar_arrive(ptx::smem_u32(&bars[4]));
        abort_flag = 0;
    }
    __syncthreads();
    const unsigned long long t0 = ptx::globaltimer_ns();
    bool ok;
    if (warp < 4) ok = ptx::mbar_wait_limit(ptx::smem_u32(&bars[warp]), 0, &abort_flag, warp == 0 ? limit_ns : ptx::WAIT_LIMIT_NS);
    else if (warp == 4) ok = wait_count(&selftest_counter, 1, &abort_flag, ptx::WAIT_LIMIT_NS);      // the wait of the tile folding: released by the flag
    else ok = ptx::mbar_wait_warp(ptx::smem_u32(&bars[lane & 1 ? 3 : 4]), 0, &abort_flag);
    const unsigned long long t1 = ptx::globaltimer_ns();
    if (warp == 5) {
        if (ok) atomicOr(err, ERR_BAD_ITEM);
    } else if (!ok && lane == 0) {
        atomicOr(err, warp == 0 ? ERR_WAIT_PRODUCER : warp == 1 ? ERR_WAIT_DEQUANT : warp == 2 ? ERR_WAIT_MMA : warp == 3 ? ERR_WAIT_SOFTMAX : ERR_WAIT_FOLD);
        waited_ns[warp] = t1 - t0;
    }
    __syncthreads();
    // and the counter wait running out by itself, with the short limit
    if (warp == 4) {
        abort_flag = 0;
        __syncwarp();
        const unsigned long long t2 = ptx::globaltimer_ns();
        const bool ok2 = wait_count(&selftest_counter, 1, &abort_flag, limit_ns);
        if (!ok2 && lane == 0) waited_ns[5] = ptx::globaltimer_ns() - t2;
    }
}
}  // namespace llattn

extern "C" int llattn_wait_selftest(unsigned long long limit_ns, int* err_word, unsigned long long* waited_ns6, void* stream) {
    if (!err_word || !waited_ns6) return fail(LLATTN_EINVAL, "wait_selftest: null pointer");
    if (limit_ns == 0 || limit_ns > 100000000ull) return fail(LLATTN_EINVAL, "wait_selftest: limit of %llu ns; 1 ns .. 100 ms", limit_ns);
    llattn::wait_selftest_kernel<<<1, 192, 0, as_stream(stream)>>>(limit_ns, err_word, waited_ns6);
    CU(cudaGetLastError());
    return LLATTN_OK;
}

#ifdef LLATTN_TRACE
// Tuning builds only: points the kernel's timeline hooks at a device buffer of 20 * 2048 64-bit words (2048 events for each of up to 20 warps).
extern "C" int llattn_debug_set_trace(void* dev_ptr) {
    CU(cudaMemcpyToSymbol(llattn::g_trace_buf, &dev_ptr, sizeof(dev_ptr)));
    return LLATTN_OK;
}
#endif
