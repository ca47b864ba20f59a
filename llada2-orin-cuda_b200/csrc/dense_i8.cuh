// Dense W4.A8 projection with residual add.
//
// It consumes the int8 activations the attention epilogue writes (values in fragment order inside every 128-group, one
// fp32 scale and one int32 sum per token and group) and the reference's 4-bit weight strips as the engine holds them on
// the device, and computes what the reference's attention-output projection computes (engine/engine.cu:434,
// moe8::gemm<.., MODE 2>, engine/moe_i8.cu:295-400), for any number of tokens:
//     Y[n][r] += sum over 128-groups g, in order, of  (s_w[r][g] * s_x[n][g]) * float(P[r][n][g] - z[r][g] * Sxq[n][g])
// with P the exact integer dot product of the group. Every float operation is the reference's (one fp32 product of
// the two scales, one fused multiply-add per group, groups in ascending order, one add into Y), so results are
// bit-identical to the reference kernel.
//
// Weight strip (16 rows x K), device layout of the reference (engine/moe_i8.cu:34-41): the 1024-byte code tiles of
// the strip's K/128 groups, then their 48-byte metas. In a code tile lane l = 4 g + t of the reference's warp owns
// bytes 16 l .. 16 l + 15 and 512 + 16 l ..: eight words; word w (step j = w / 2, half h = w % 2) holds, for k = 32 j +
// 16 h + 4 t + e (e = byte index), the code of row g in the low nibble and of row g + 8 in the high nibble
// (engine/moe_i8.cu:127-160). A meta holds fp16 scale pairs (rows g | g + 8) at 4 g and zero-point pairs at 32 + 2 g.
//
// The first two kernels use mma.sync m16n8k32 (u8 x s8 -> s32), whose fragments these layouts are: a lane's eight code words ARE its
// A fragments (one nibble mask per register) and a token's B fragments are 32 contiguous bytes per lane, so operands go
// from memory to the tensor core without being unpacked into shared memory, and the integers come out in registers,
// where the fold into fp32 needs them. What the path costs is that fold, 16 float steps per output which cannot be
// reordered, not the products.
//   dense_strip_kernel  a decode step's few tokens: a CTA takes ONE strip and one warp per 128-group works on it; the
//                       integers of all groups exist at once, only the multiply-adds run in group order.
//   dense_tile_kernel   many tokens: 128 rows x 16, 32 or 64 tokens per CTA.
//   dense_wide_kernel   more tokens, or more groups: 128 rows x 32, 64 or 128 tokens per CTA, the products on tcgen05 (kind::i8).
#pragma once
#include <cuda_fp16.h>
#include "common.cuh"
#include "ptx.cuh"

namespace llattn {

constexpr int DN_ROWS = 128, DN_GROUP = 128;
constexpr int DN_TILE_BYTES = 1024, DN_META_BYTES = 48;

struct DenseParams {
    const uint8_t* W;      // strips
    const int8_t* q;       // [ntokens][K], fragment order inside every 128-group
    const float* s;        // [ntokens][K / 128]
    const int32_t* sum;    // [ntokens][K / 128]
    float* Y;              // [ntokens][rows], accumulated into
    int ntokens, rows, K;
    int* err;              // the caller's device error word, or null: the library's own
};

// What calls without an error word of their own report in: one word per device, part of the library image, read and cleared by
// llattn_dense_status. (Not in an allocation: a first call may be under stream capture.)
static __device__ int g_dense_err;
__device__ __forceinline__ void report_error(const DenseParams& p, int bits) { atomicOr(p.err ? p.err : &g_dense_err, bits); }

__device__ __forceinline__ void mma_m16n8k32_u8s8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// int -> float through the float whose bits are 1.5 * 2^23 + v: exact for |v| < 2^22 (here |v| <= 255 * 127 * 128). An
// integer add and a float subtract at full rate; the conversion instruction has an eighth of it.
__device__ __forceinline__ float small_int_to_float(int v) { return __int_as_float(v + 0x4B400000) - 12582912.0f; }

// ------------------------------------------------------------------------------------------------------------- few tokens
// Bound by latency: 2.2 MB of weights are 0.34 us of HBM time and 32 tokens x 2048 x 2048 are nothing, so what counts is
// the length of the dependent chain and how many SMs pull on the weights: one CTA per (strip, 32 tokens), 128 CTAs at
// 2048 rows, warp w on group w (w + 16, ... when K > 2048). Each warp leaves the two factors of its group's multiply-add
// in shared memory; then thread = output element runs the sixteen in order.
// Measured, 2048 x 2048, launches in a graph over 20 different weights: 32 tokens 4.0 us (a 128-row tile per CTA, group after group: 17.7),
// 1 token 2.7 us (17.3).
constexpr int DS_WARPS = 16, DS_THREADS = 32 * DS_WARPS, DS_TOK = 32;
constexpr int DS_LD = 18;                          // (value, scale) pairs per token row of 16: keeps the fragment writes conflict-free
constexpr int DS_SMEM_BYTES = DS_WARPS * DS_TOK * DS_LD * 8;

__global__ void __launch_bounds__(DS_THREADS, 1) dense_strip_kernel(const DenseParams p) {
    extern __shared__ __align__(16) uint8_t ds_smem[];
    ptx::grid_dependency_wait();               // nothing is read or written before the kernel ahead has completed
    float2* pairs = reinterpret_cast<float2*>(ds_smem);               // [warp][token][DS_LD]: (float of the integer, s_w * s_x)
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int strip = blockIdx.x, n0 = blockIdx.y * DS_TOK, live = min(DS_TOK, p.ntokens - n0);
    const int ktot = p.K / DN_GROUP;
    const uint8_t* codes = p.W + size_t(strip) * ktot * (DN_TILE_BYTES + DN_META_BYTES);
    const uint8_t* metas = codes + size_t(ktot) * DN_TILE_BYTES;
    // this thread's output element: row tid % 16 of the strip, token tid / 16; its old value is on its way from the start
    const int row = tid & 15, tok = tid >> 4;
    float* yp = p.Y + size_t(n0 + tok) * p.rows + strip * 16 + row;
    float y = 0.f, c = 0.f;
#pragma unroll 1
    for (int k0 = 0; k0 < ktot; k0 += DS_WARPS) {
        const int gi = k0 + warp;
        if (gi < ktot) {
            const uint4 lo = __ldg(reinterpret_cast<const uint4*>(codes + size_t(gi) * DN_TILE_BYTES + 16 * lane));
            const uint4 hi = __ldg(reinterpret_cast<const uint4*>(codes + size_t(gi) * DN_TILE_BYTES + 512 + 16 * lane));
            const uint32_t sw2 = __ldg(reinterpret_cast<const uint32_t*>(metas + size_t(gi) * DN_META_BYTES + 4 * g));
            const uint32_t z2 = __ldg(reinterpret_cast<const uint16_t*>(metas + size_t(gi) * DN_META_BYTES + 32 + 2 * g));
            uint4 b[4][2];
            float sx[4][2];
            int sq[4][2];
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                const int n = 8 * nt + g;
                b[nt][0] = b[nt][1] = make_uint4(0u, 0u, 0u, 0u);
                if (n < live) {
                    const uint4* src = reinterpret_cast<const uint4*>(p.q + size_t(n0 + n) * p.K + size_t(gi) * DN_GROUP + 32 * t);
                    b[nt][0] = __ldg(src);
                    b[nt][1] = __ldg(src + 1);
                }
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const size_t at = size_t(n0 + min(8 * nt + 2 * t + e, live - 1)) * ktot + gi;
                    sx[nt][e] = __ldg(p.s + at);
                    sq[nt][e] = __ldg(p.sum + at);
                }
            }
            if (k0 == 0 && tok < live) y = __ldcg(yp);
            const uint32_t w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
            const uint32_t mk = 0x0F0F0F0Fu;
            const float swa = __half2float(__ushort_as_half(uint16_t(sw2 & 0xffffu))), swb = __half2float(__ushort_as_half(uint16_t(sw2 >> 16)));
            const int za = int(z2 & 0xffu), zb = int(z2 >> 8);
            float2* out = pairs + warp * DS_TOK * DS_LD;
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                if (8 * nt >= live) break;
                int acc[4] = {0, 0, 0, 0};
                const uint32_t bw[8] = {b[nt][0].x, b[nt][0].y, b[nt][0].z, b[nt][0].w, b[nt][1].x, b[nt][1].y, b[nt][1].z, b[nt][1].w};
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    mma_m16n8k32_u8s8(acc, w[2 * j] & mk, (w[2 * j] >> 4) & mk, w[2 * j + 1] & mk, (w[2 * j + 1] >> 4) & mk, bw[2 * j], bw[2 * j + 1]);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    float2* o = out + (8 * nt + 2 * t + e) * DS_LD + g;
                    o[0] = make_float2(small_int_to_float(acc[e] - za * sq[nt][e]), __fmul_rn(swa, sx[nt][e]));
                    o[8] = make_float2(small_int_to_float(acc[2 + e] - zb * sq[nt][e]), __fmul_rn(swb, sx[nt][e]));
                }
            }
        } else if (k0 == 0 && tok < live) {
            y = __ldcg(yp);
        }
        __syncthreads();
        if (tok < live) {
            const int ng = min(DS_WARPS, ktot - k0);
            const float2* in = pairs + tok * DS_LD + row;
#pragma unroll 16
            for (int k = 0; k < ng; ++k) {
                const float2 vs = in[k * DS_TOK * DS_LD];
                c = __fmaf_rn(vs.y, vs.x, c);
            }
        }
        if (k0 + DS_WARPS < ktot) __syncthreads();
    }
    if (tok < live) __stcg(yp, y + c);
}

// ------------------------------------------------------------------------------------------------------------ many tokens
// CTA = 128 rows x TOK (16, 32 or 64) tokens, 8 warps of 32 rows x TOK / 2 tokens. Everything a group needs comes in through cp.async, DT_STAGES - 1
// groups ahead: the strips' codes and metas, the tokens' codes, scales and sums (16-byte
// chunk c of token n at chunk position c ^ (n % 8): conflict-free fragment loads). Then two strips' MMAs, all output tiles in
// turn so that a chain of four K-steps hides behind the others, and the fold of TOK / 2 outputs per thread, two per
// instruction where fp32 comes in pairs.
// What bounds it: about 200 issue slots and 32 MMAs (8.8 cycles each on a scheduler) per warp and group of 1,024 outputs -
// 2048 tokens x 2048 x 2048: 17 us of tensor pipe over 148 SMs - then reading and writing Y (33.6 MB, 5.1 us; brought
// into L2 while the groups run).
// Measured, 2048 x 2048, launches in a graph: 2048 tokens 51 us (a warp per strip and 64 tokens, whose
// fragment loads took half of the shared-memory bandwidth: 4 more; the tcgen05 form it replaces: 60), 128 tokens 8.5 us (16-token
// tiles; 16.4 with 64).
constexpr int DT_THREADS = 256, DT_STAGES = 4;
template <int TOK> struct DenseTile {                              // shared-memory layout of a stage: codes, q, scales, sums, metas
    static constexpr int Q = 8 * DN_TILE_BYTES, SX = Q + TOK * 128, SQ = SX + TOK * 4, META = SQ + TOK * 4, STAGE = META + 8 * DN_META_BYTES;
    static constexpr int SMEM = DT_STAGES * STAGE, NT = TOK / 16;  // NT: 8-token output tiles per warp and strip
};

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(uint32_t a, uint32_t b) { f32x2 d; asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(a), "r"(b)); return d; }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) { f32x2 d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) { f32x2 d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ f32x2 fma2v(f32x2 a, f32x2 b, f32x2 c) { f32x2 d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }

// 16- and 4-byte asynchronous copies global -> shared (per-thread completion groups); `live` false writes zeros.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool live) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src, bool live) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(live ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kPending> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(kPending) : "memory"); }

template <int TOK>
__global__ void __launch_bounds__(DT_THREADS, TOK == 64 ? 2 : 3) dense_tile_kernel(const DenseParams p) {
    using T = DenseTile<TOK>;
    extern __shared__ __align__(128) uint8_t dt_smem[];
    ptx::grid_dependency_wait();               // nothing is read or written before the kernel ahead has completed
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int row0 = blockIdx.x * DN_ROWS, n0 = blockIdx.y * TOK, live = min(TOK, p.ntokens - n0);
    const int ktot = p.K / DN_GROUP;
    const uint8_t* codes = p.W + size_t((row0 >> 4) + warp) * ktot * (DN_TILE_BYTES + DN_META_BYTES);
    const uint8_t* metas = codes + size_t(ktot) * DN_TILE_BYTES;
    const uint32_t sm0 = ptx::smem_u32(dt_smem);
    // this thread's part of a stage: its lane's code words, one of the strip's three meta chunks, chunk tid % 8 of tokens
    // tid / 8 and tid / 8 + 32, and one scale or sum
    const int cn = tid >> 3, cc = tid & 7;
    const int8_t* src = p.q + size_t(n0 + min(cn, live - 1)) * p.K + 16 * cc;
    const int8_t* src32 = p.q + size_t(n0 + min(cn + 32, live - 1)) * p.K + 16 * cc;
    const uint32_t dst0 = sm0 + T::Q + cn * 128 + ((cc ^ (cn & 7)) << 4);
    const int sn = tid & (TOK - 1);
    const size_t sat = size_t(n0 + min(sn, live - 1)) * ktot;
    const void* ssrc = tid < TOK ? static_cast<const void*>(p.s + sat) : static_cast<const void*>(p.sum + sat);
    const uint32_t sdst = sm0 + T::SX + 4 * (tid & (2 * TOK - 1));
    auto fetch = [&](int i) {                  // one commit per call, so groups count uniformly
        if (i < ktot) {
            const uint32_t st = uint32_t(i % DT_STAGES) * T::STAGE;
            const uint32_t mine = sm0 + warp * DN_TILE_BYTES + 16 * lane + st;
            cp_async16(mine, codes + size_t(i) * DN_TILE_BYTES + 16 * lane, true);
            cp_async16(mine + 512, codes + size_t(i) * DN_TILE_BYTES + 512 + 16 * lane, true);
            if (lane < 3) cp_async16(sm0 + T::META + warp * DN_META_BYTES + 16 * lane + st, metas + size_t(i) * DN_META_BYTES + 16 * lane, true);
            if (TOK >= 32 || cn < TOK) cp_async16(dst0 + st, src + size_t(i) * DN_GROUP, cn < live);
            if (TOK == 64) cp_async16(dst0 + st + 32 * 128, src32 + size_t(i) * DN_GROUP, cn + 32 < live);
            if (tid < 2 * TOK) cp_async4(sdst + st, static_cast<const uint8_t*>(ssrc) + 4 * size_t(i), sn < live);
        }
        cp_async_commit();
    };
    for (int i = 0; i < DT_STAGES - 1; ++i) fetch(i);
    // the tile's TOK x 512 bytes of Y into L2: wanted when the last group is folded
    if ((tid >> 2) < live) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.Y + size_t(n0 + (tid >> 2)) * p.rows + row0 + 32 * (tid & 3)));
    // this warp: strips 2 (warp / 2) and + 1, tokens TOK / 2 (warp % 2) .. + TOK / 2 - 1
    const int sp = 2 * (warp >> 1), tb = TOK / 2 * (warp & 1);
    f32x2 c[2][T::NT][2];                          // per strip and n-tile: rows g and g + 8, tokens tb + 8 nt + 2 t and + 1
#pragma unroll
    for (int k = 0; k < 4 * T::NT; ++k) (&c[0][0][0])[k] = 0ull;
    const f32x2 magic = 0xCB400000CB400000ull; // -1.5 * 2^23 twice
#pragma unroll 1
    for (int i = 0; i < ktot; ++i) {
        cp_async_wait<DT_STAGES - 2>();
        __syncthreads();                       // group i is in for everybody; group i - 1 is done with, its stage can be refilled
        fetch(i + DT_STAGES - 1);
        const uint8_t* st = dt_smem + (i % DT_STAGES) * T::STAGE;
        uint32_t w[2][8];                      // the lane's code words of both strips
        float swa[2], swb[2];
        int za[2], zb[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const uint8_t* meta = st + T::META + (sp + u) * DN_META_BYTES;
            const uint32_t sw2 = *reinterpret_cast<const uint32_t*>(meta + 4 * g), z2 = *reinterpret_cast<const uint16_t*>(meta + 32 + 2 * g);
            swa[u] = __half2float(__ushort_as_half(uint16_t(sw2 & 0xffffu))); swb[u] = __half2float(__ushort_as_half(uint16_t(sw2 >> 16)));
            za[u] = int(z2 & 0xffu); zb[u] = int(z2 >> 8);
            *reinterpret_cast<uint4*>(&w[u][0]) = *reinterpret_cast<const uint4*>(st + (sp + u) * DN_TILE_BYTES + 16 * lane);
            *reinterpret_cast<uint4*>(&w[u][4]) = *reinterpret_cast<const uint4*>(st + (sp + u) * DN_TILE_BYTES + 512 + 16 * lane);
        }
        const uint32_t mk = 0x0F0F0F0Fu;
        int acc[2][T::NT][4] = {};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            uint4 b[T::NT];
#pragma unroll
            for (int k = 0; k < T::NT; ++k) b[k] = *reinterpret_cast<const uint4*>(st + T::Q + (tb + 8 * k + g) * 128 + (((2 * t + h) ^ g) << 4));
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const uint32_t x = w[u][4 * h + 2 * j], y = w[u][4 * h + 2 * j + 1], a0 = x & mk, a1 = (x >> 4) & mk, a2 = y & mk, a3 = (y >> 4) & mk;
#pragma unroll
                    for (int k = 0; k < T::NT; ++k) mma_m16n8k32_u8s8(acc[u][k], a0, a1, a2, a3, j ? b[k].z : b[k].x, j ? b[k].w : b[k].y);
                }
        }
#pragma unroll
        for (int k = 0; k < T::NT; ++k) {
            const f32x2 sx = *reinterpret_cast<const f32x2*>(st + T::SX + 4 * tb + 8 * t + 32 * k);
            const int2 sq = *reinterpret_cast<const int2*>(st + T::SQ + 4 * tb + 8 * t + 32 * k);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const f32x2 va = add2(pack2(uint32_t(acc[u][k][0] + (0x4B400000 - za[u] * sq.x)), uint32_t(acc[u][k][1] + (0x4B400000 - za[u] * sq.y))), magic);
                const f32x2 vb = add2(pack2(uint32_t(acc[u][k][2] + (0x4B400000 - zb[u] * sq.x)), uint32_t(acc[u][k][3] + (0x4B400000 - zb[u] * sq.y))), magic);
                c[u][k][0] = fma2v(mul2(pack2(__float_as_uint(swa[u]), __float_as_uint(swa[u])), sx), va, c[u][k][0]);
                c[u][k][1] = fma2v(mul2(pack2(__float_as_uint(swb[u]), __float_as_uint(swb[u])), sx), vb, c[u][k][1]);
            }
        }
    }
    cp_async_wait<0>();
    // Y += c: a warp's access covers the 8 rows of four tokens, whole 32-byte sectors
    float* ybase = p.Y + size_t(n0 + tb + 2 * t) * p.rows + row0 + 16 * sp + g;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        float y[T::NT][4];
#pragma unroll
        for (int k = 0; k < T::NT; ++k)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                y[k][e] = tb + 8 * k + 2 * t + (e & 1) < live ? __ldcg(ybase + size_t(8 * k + (e & 1)) * p.rows + 16 * u + 8 * (e >> 1)) : 0.f;
#pragma unroll
        for (int k = 0; k < T::NT; ++k)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (tb + 8 * k + 2 * t + (e & 1) < live) {
                    const f32x2 v = c[u][k][e >> 1];
                    __stcg(ybase + size_t(8 * k + (e & 1)) * p.rows + 16 * u + 8 * (e >> 1), y[k][e] + __uint_as_float(uint32_t(e & 1 ? v >> 32 : v)));
                }
    }
}

// ------------------------------------------------------------------------------------------------------- very many tokens
// Tiles of 128 rows x N tokens, one CTA per SM that walks its share of them, the products on tcgen05 kind::i8 (u8 x s8, M = 128; 74 cycles for
// 128 x 128 x 32 of them, where mma.sync takes 8.8 for 16 x 8 x 32 on each of four schedulers, both measured: 3.8 times the rate), so that
// the fold is what is left: sixteen warps, six instructions per two outputs and group. The other roles run ahead of them, into the next
// tile too, through rings whose slots hold TWO groups: a warp by itself issues an instruction every five cycles or so, and with a slot per
// group the barriers' instructions alone took a role 1,500 cycles a group.
//   producer warp  bulk copies of the strips' codes into a ring, 2 KB a copy
//   unpack warps   codes -> u8 rows in the 128-byte-swizzle operand layout
//   load warps     activations, cp.async straight into the operand layout (completion by mbarrier, no waiting)
//   MMA warp       four K-steps a group into one of four accumulators
// The factors of the fold (token scales and sums, row scales and zero points) of sixteen groups lie in shared memory as floats.
// Measured, 2048 x 2048, launches in a graph, mma.sync tiles / a CTA per tile, two rounds of accumulators a group / this: 320 tokens 16.7 /
// 11.8 / 11.7 us, 640 26.5 / 17.4 / 16.5, 1024 26.0 / 17.7 / 16.8, 2048 49.7 / 34.3 / 30.6, 4096 - / 67.7 / 58.5. A tile of 128 tokens takes 0.68 us a
// group, 56 % of the issue slots and 42 % of the fp32 pipe over the kernel; its start and end are 6 us for a CTA's first and 3 for the others.
constexpr int DW_FOLD_WARPS = 16, DW_UNPACK_WARPS = 4, DW_LOAD_WARPS = 2;
constexpr int DW_WARP_UNPACK = DW_FOLD_WARPS, DW_WARP_LOAD = DW_WARP_UNPACK + DW_UNPACK_WARPS, DW_WARP_PRODUCER = DW_WARP_LOAD + DW_LOAD_WARPS,
              DW_WARP_MMA = DW_WARP_PRODUCER + 1, DW_THREADS = 32 * (DW_WARP_MMA + 1);
// Registers a thread: at launch, and after the roles have parted. The second split has to come out of the first, or its waits for registers
// would not end; that the compiler gave each kernel the first number is checked before the first launch, and without it the tiles take the call.
#ifndef LLATTN_DW_LAUNCH_REGS
#define LLATTN_DW_LAUNCH_REGS 80
#endif
constexpr int DW_LAUNCH_REGS = LLATTN_DW_LAUNCH_REGS, DW_FOLD_REGS = 96, DW_OTHER_REGS = 48;
static_assert(DW_FOLD_WARPS * DW_FOLD_REGS + (DW_THREADS / 32 - DW_FOLD_WARPS) * DW_OTHER_REGS <= DW_THREADS / 32 * DW_LAUNCH_REGS && DW_THREADS % 128 == 0 &&
              DW_FOLD_WARPS % 4 == 0, "register split");
constexpr int DW_RAW = 2, DW_A = 2, DW_B = 2, DW_ACC = 4, DW_SC = 16;      // ring slots; groups of factors held
template <int N> struct DenseWide {
    static constexpr int A_GROUP = DN_ROWS * DN_GROUP, B_GROUP = N * DN_GROUP, RAW_GROUP = 8 * DN_TILE_BYTES;
    static constexpr int A = 0, B = A + DW_A * 2 * A_GROUP, RAW = B + DW_B * 2 * B_GROUP;
    static constexpr int LD_T = N + 4, LD_R = DN_ROWS + 1;                 // a group's token factors and rows, padded for the transposing stores
    static constexpr int SX = RAW + DW_RAW * 2 * RAW_GROUP, SQ = SX + DW_SC * LD_T * 4, WZ = SQ + DW_SC * LD_T * 4;
    static constexpr int BAR = WZ + DW_SC * LD_R * 8, SMEM = BAR + 8 * 32;
    static constexpr int COLS = N / 4;                                     // a fold warp's tokens
    static constexpr int TMEM = DW_ACC * N;
};
enum { WB_RAW_FULL = 0, WB_RAW_EMPTY = WB_RAW_FULL + DW_RAW, WB_A_FULL = WB_RAW_EMPTY + DW_RAW, WB_A_EMPTY = WB_A_FULL + DW_A,
       WB_B_FULL = WB_A_EMPTY + DW_A, WB_B_EMPTY = WB_B_FULL + DW_B, WB_ACC_FULL = WB_B_EMPTY + DW_B, WB_ACC_EMPTY = WB_ACC_FULL + DW_ACC,
       WB_SC_FULL = WB_ACC_EMPTY + DW_ACC, WB_SC_EMPTY, WB_SPARE, WB_COUNT };
static_assert(WB_COUNT <= 32, "barrier area");

// kind::i8 instruction descriptor: s32 accumulator, A u8 (format 0), B s8 (format 1), both K-major.
__host__ __device__ constexpr uint32_t idesc_i8_u8s8(int M, int N) {
    return (2u << 4) | (0u << 7) | (1u << 10) | (uint32_t(N >> 3) << 17) | (uint32_t(M >> 4) << 24);
}
// A group: four K-steps of 32 over 128-byte-swizzle tiles, the first overwriting the accumulator, and a commit.
__device__ __forceinline__ void mma_i8_group_warp(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc, uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred pe, pf, pt;\n\t.reg .b32 x, y;\n\t.reg .b64 da, db;\n\t"
        "elect.sync _|pe, 0xffffffff;\n\t"
        "setp.ne.b32 pf, 0, 0;\n\t setp.eq.b32 pt, 0, 0;\n\t"
        "mov.b64 da, {%1, %3};\n\t mov.b64 db, {%2, %3};\n\t"
        "@pe tcgen05.mma.cta_group::1.kind::i8 [%0], da, db, %4, pf;\n\t"
        "add.u32 x, %1, 2;\n\t add.u32 y, %2, 2;\n\t mov.b64 da, {x, %3};\n\t mov.b64 db, {y, %3};\n\t"
        "@pe tcgen05.mma.cta_group::1.kind::i8 [%0], da, db, %4, pt;\n\t"
        "add.u32 x, %1, 4;\n\t add.u32 y, %2, 4;\n\t mov.b64 da, {x, %3};\n\t mov.b64 db, {y, %3};\n\t"
        "@pe tcgen05.mma.cta_group::1.kind::i8 [%0], da, db, %4, pt;\n\t"
        "add.u32 x, %1, 6;\n\t add.u32 y, %2, 6;\n\t mov.b64 da, {x, %3};\n\t mov.b64 db, {y, %3};\n\t"
        "@pe tcgen05.mma.cta_group::1.kind::i8 [%0], da, db, %4, pt;\n\t"
        "@pe tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%5];\n\t"
        "}\n" :: "r"(d), "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"(bar) : "memory");
}
// An arrival on `bar` once this thread's cp.async so far have landed.
__device__ __forceinline__ void cp_async_arrive(uint32_t bar) { asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory"); }

template <int N, bool ONE>
__global__ void __launch_bounds__(DW_THREADS, 1) dense_wide_kernel(const DenseParams p) {
    using T = DenseWide<N>;
    extern __shared__ __align__(1024) uint8_t dw_smem[];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_word;
    volatile int* const abort_flag = &abort_word;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ktot = p.K / DN_GROUP, nst = (ktot + 1) / 2;       // stages: two groups each, the last one perhaps a single one
    const int row_tiles = p.rows / DN_ROWS, tiles = row_tiles * ((p.ntokens + N - 1) / N);
    // ONE: a grid of row tiles x token tiles, a CTA each, which needs no divisions on its way
    auto row_tile = [&](int tile) -> int { return ONE ? int(blockIdx.x) : tile % row_tiles; };
    auto token_tile = [&](int tile) -> int { return ONE ? int(blockIdx.y) : tile / row_tiles; };
    const uint32_t sm0 = ptx::smem_u32(dw_smem), bar0 = sm0 + T::BAR;
    auto BAR = [&](int i) -> uint32_t { return bar0 + 8u * uint32_t(i); };
    if (sm0 & 1023u) {                         // the swizzled tiles need a 1024-byte aligned base: report, do nothing
        ptx::grid_dependency_wait();           // and let no kernel behind this one start before the one ahead has completed
        if (tid == 0) report_error(p, ERR_SMEM_ALIGN);
        return;
    }
    if (tid == 0) {
        for (int i = 0; i < DW_RAW; ++i) { ptx::mbar_init(BAR(WB_RAW_FULL + i), 1); ptx::mbar_init(BAR(WB_RAW_EMPTY + i), 32 * DW_UNPACK_WARPS); }
        for (int i = 0; i < DW_A; ++i) { ptx::mbar_init(BAR(WB_A_FULL + i), 32 * DW_UNPACK_WARPS); ptx::mbar_init(BAR(WB_A_EMPTY + i), 1); }
        for (int i = 0; i < DW_B; ++i) { ptx::mbar_init(BAR(WB_B_FULL + i), 32 * DW_LOAD_WARPS); ptx::mbar_init(BAR(WB_B_EMPTY + i), 1); }
        for (int i = 0; i < DW_ACC; ++i) { ptx::mbar_init(BAR(WB_ACC_FULL + i), 1); ptx::mbar_init(BAR(WB_ACC_EMPTY + i), 32 * DW_FOLD_WARPS); }
        ptx::mbar_init(BAR(WB_SC_FULL), 32 * DW_FOLD_WARPS); ptx::mbar_init(BAR(WB_SC_EMPTY), 32 * DW_FOLD_WARPS);
        ptx::mbar_init(BAR(WB_SPARE), 1);
        ptx::fence_mbar_init();
        abort_word = 0;
    }
    if (warp == DW_WARP_MMA) { ptx::tmem_alloc(ptx::smem_u32(&tmem_slot), T::TMEM); ptx::tmem_relinquish(); }
    ptx::grid_dependency_wait();               // nothing is read or written before the kernel ahead has completed
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const size_t strip_bytes = size_t(ktot) * (DN_TILE_BYTES + DN_META_BYTES);
    int errbits = 0;
    // Wait for use `u` of a slot to be filled / for the previous use of a slot to be over (the first needs no wait). The roles that go on to
    // warp-wide instructions take the form with one answer per warp. Its votes cost 1 to 1.5 % (2048 x 2048, 2048 tokens 34.6 -> 35.0 us);
    // lanes that give up but walk on with their warp, arriving nowhere, cost more (36.3).
    auto filled = [&](int bar, int u, int err) -> bool {
        if (ptx::mbar_wait(BAR(bar), u & 1, abort_flag)) return true;
        errbits |= err;
        return false;
    };
    auto emptied = [&](int bar, int u, int err) -> bool { return u == 0 || filled(bar, u - 1, err); };
    auto filled_warp = [&](int bar, int u, int err) -> bool {
        if (ptx::mbar_wait_warp(BAR(bar), u & 1, abort_flag)) return true;
        errbits |= err;
        return false;
    };
    auto emptied_warp = [&](int bar, int u, int err) -> bool { return u == 0 || filled_warp(bar, u - 1, err); };

    // The folding warps' registers come from the others: 96 take in all accumulators of a group at once (with 80, and two rounds of 16 of the
    // 32, a tile of 128 x 128 x 2048 took 17.7 us, now 16.8; one of 64 tokens 12.5 and 11.7).
    if (warp < DW_FOLD_WARPS) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(DW_FOLD_REGS));
    else asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(DW_OTHER_REGS));
    if (warp < DW_FOLD_WARPS) {
        // ---- fold: a warp has 32 rows and COLS tokens, as an mma fragment: lane l rows l / 4 + 8 k, tokens 8 i + 2 (l % 4) and + 1. Two token
        // factors then serve eight outputs (with a row a lane: two).
        constexpr int C = T::COLS;
        const int row = 32 * (warp & 3) + (lane >> 2), col = C * (warp >> 2) + 2 * (lane & 3);
        const uint32_t tacc = tmem + (uint32_t(32 * (warp & 3)) << 16) + C * (warp >> 2);
        float* const sx = reinterpret_cast<float*>(dw_smem + T::SX);
        float* const sq = reinterpret_cast<float*>(dw_smem + T::SQ);
        float2* const wz = reinterpret_cast<float2*>(dw_smem + T::WZ);
        f32x2 c[C / 8][4];                             // per eight tokens: rows row, + 8, + 16, + 24
        const f32x2 magic = 0xCB400000CB400000ull;     // -1.5 * 2^23 twice
        bool alive = true;
        int u = 0, ga = 0;                             // blocks of factors and groups so far, over all tiles
#pragma unroll 1
        for (int tile = blockIdx.x; tile < tiles && alive; tile += ONE ? tiles : int(gridDim.x)) {
            const int row0 = row_tile(tile) * DN_ROWS, n0 = token_tile(tile) * N, live = min(N, p.ntokens - n0);
            const uint8_t* strips = p.W + size_t(row0 >> 4) * strip_bytes;
#pragma unroll
            for (int j = 0; j < C / 2; ++j) (&c[0][0])[j] = 0ull;
#pragma unroll 1
            for (int g0 = 0; g0 < ktot && alive; g0 += DW_SC, ++u) {
                // the factors of the next sixteen groups: thread = (token or row, group)
                if (!emptied_warp(WB_SC_EMPTY, u, ERR_WAIT_SOFTMAX)) { alive = false; break; }
                const int g = tid & 15, gi = min(g0 + g, ktot - 1);
#pragma unroll
                for (int k = 0; k < (N + 31) / 32; ++k) {
                    const int n = (tid >> 4) + 32 * k;
                    const size_t at = size_t(n0 + min(n, live - 1)) * ktot + gi;
                    sx[g * T::LD_T + n] = __ldg(p.s + at);
                    sq[g * T::LD_T + n] = float(__ldg(p.sum + at));
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int r = (tid >> 4) + 32 * k, rr = r & 15;
                    const uint8_t* mt = strips + size_t(r >> 4) * strip_bytes + size_t(ktot) * DN_TILE_BYTES + size_t(gi) * DN_META_BYTES;
                    wz[g * T::LD_R + r] = make_float2(__half2float(__ushort_as_half(__ldg(reinterpret_cast<const uint16_t*>(mt + 4 * (rr & 7) + 2 * (rr >> 3))))),
                                                      -float(__ldg(mt + 32 + 2 * (rr & 7) + (rr >> 3))));
                }
                ptx::mbar_arrive(BAR(WB_SC_FULL));
                if (!filled_warp(WB_SC_FULL, u, ERR_WAIT_SOFTMAX)) { alive = false; break; }
                const int ng = min(DW_SC, ktot - g0);
#pragma unroll 1
                for (int i = 0; i < ng; ++i, ++ga) {
                    const int slot = ga % DW_ACC;
                    f32x2 sw[4], nz[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const float2 f = wz[i * T::LD_R + row + 8 * k];
                        sw[k] = pack2(__float_as_uint(f.x), __float_as_uint(f.x)); nz[k] = pack2(__float_as_uint(f.y), __float_as_uint(f.y));
                    }
                    if (!filled_warp(WB_ACC_FULL + slot, ga / DW_ACC, ERR_WAIT_SOFTMAX)) { alive = false; break; }
                    ptx::tc_fence_after();
                    uint32_t d0[C / 2], d1[C / 2];     // rows + 0, + 8 and rows + 16, + 24
                    ptx::tmem_ld16x256_cols(tacc + slot * N, d0);
                    ptx::tmem_ld16x256_cols(tacc + slot * N + (16u << 16), d1);
                    ptx::tmem_wait_ld_tied(d0);
                    ptx::tmem_wait_ld_tied(d1);
                    ptx::tc_fence_before();
                    ptx::mbar_arrive(BAR(WB_ACC_EMPTY + slot));
#pragma unroll
                    for (int j = 0; j < C / 8; ++j) {
                        const f32x2 x = *reinterpret_cast<const f32x2*>(sx + i * T::LD_T + col + 8 * j), q = *reinterpret_cast<const f32x2*>(sq + i * T::LD_T + col + 8 * j);
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const uint32_t *d = (k < 2 ? d0 : d1) + 4 * j + 2 * (k & 1);
                            // float(P - z sq) = (1.5 * 2^23 + P) + (-z sq - 1.5 * 2^23): both terms are whole numbers below 2^24 in
                            // magnitude (|P|, |z sq| <= 255 * 128 * 128 = 4,177,920), so every step is exact
                            const f32x2 v = add2(pack2(d[0] + 0x4B400000u, d[1] + 0x4B400000u), fma2v(nz[k], q, magic));
                            c[j][k] = fma2v(mul2(sw[k], x), v, c[j][k]);
                        }
                    }
                }
                ptx::mbar_arrive(BAR(WB_SC_EMPTY));
            }
            if (alive) {
                // Y += c: a warp's access is eight rows of four tokens, whole sectors; all loads before the first add
                float* y0 = p.Y + size_t(n0 + col) * p.rows + row0 + row;
                float y[C / 8][4][2];
#pragma unroll
                for (int j = 0; j < C / 8; ++j)
#pragma unroll
                    for (int k = 0; k < 4; ++k)
#pragma unroll
                        for (int e = 0; e < 2; ++e) y[j][k][e] = col + 8 * j + e < live ? __ldcg(y0 + size_t(8 * j + e) * p.rows + 8 * k) : 0.f;
#pragma unroll
                for (int j = 0; j < C / 8; ++j)
#pragma unroll
                    for (int k = 0; k < 4; ++k)
#pragma unroll
                        for (int e = 0; e < 2; ++e)
                            if (col + 8 * j + e < live)
                                __stcg(y0 + size_t(8 * j + e) * p.rows + 8 * k, y[j][k][e] + __uint_as_float(uint32_t(e ? c[j][k] >> 32 : c[j][k])));
            }
        }
    } else if (warp < DW_WARP_LOAD) {
        // ---- unpack: this warp's two strips of every group. Word k of lane l = 4 g + t holds the codes at fragment positions
        // 32 t + 4 k .. + 3, of row g in the low nibbles and of row g + 8 in the high ones: words 0-3 are the 16-byte chunk 2 t of these
        // rows, words 4-7 chunk 2 t + 1. A quarter warp's stores cover eight chunk positions.
        const int g = lane >> 2, t = lane & 3, s0 = 2 * (warp - DW_WARP_UNPACK);
        const uint32_t m = 0x0F0F0F0Fu;
        const uint8_t* const src = dw_smem + T::RAW + s0 * 2 * DN_TILE_BYTES + 16 * lane;
        uint8_t* const dst0 = dw_smem + T::A + (16 * s0 + g) * 128 + (((2 * t) ^ g) << 4);
        uint8_t* const dst1 = dw_smem + T::A + (16 * s0 + g) * 128 + (((2 * t + 1) ^ g) << 4);
        const int total = ONE ? nst : nst * ((tiles - int(blockIdx.x) + int(gridDim.x) - 1) / int(gridDim.x));      // stages of all tiles of this CTA
#pragma unroll 1
        for (int i = 0; i < total; ++i) {
            const int b = i & 1, u = i >> 1;
            static_assert(DW_RAW == 2 && DW_A == 2 && DW_B == 2, "slot = stage % 2");
            if (!filled(WB_RAW_FULL + b, u, ERR_WAIT_DEQUANT) || !emptied(WB_A_EMPTY + b, u, ERR_WAIT_DEQUANT)) break;
#pragma unroll
            for (int e = 0; e < 2; ++e) {              // the stage's groups (a missing one is whatever the slot held: no MMA reads it)
                uint4 w[2][2];
#pragma unroll
                for (int k = 0; k < 2; ++k)
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        w[k][h] = *reinterpret_cast<const uint4*>(src + b * 2 * T::RAW_GROUP + k * 2 * DN_TILE_BYTES + e * DN_TILE_BYTES + 512 * h);
#pragma unroll
                for (int k = 0; k < 2; ++k)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        uint8_t* a = (h ? dst1 : dst0) + (2 * b + e) * T::A_GROUP + 16 * k * 128;
                        const uint4 x = w[k][h];
                        *reinterpret_cast<uint4*>(a) = make_uint4(x.x & m, x.y & m, x.z & m, x.w & m);
                        *reinterpret_cast<uint4*>(a + 8 * 128) = make_uint4((x.x >> 4) & m, (x.y >> 4) & m, (x.z >> 4) & m, (x.w >> 4) & m);
                    }
            }
            ptx::mbar_arrive(BAR(WB_RAW_EMPTY + b));
            ptx::fence_proxy_async_smem();
            ptx::mbar_arrive(BAR(WB_A_FULL + b));
        }
    } else if (warp < DW_WARP_PRODUCER) {
        // ---- activations: 16-byte chunk c of token n at chunk position c ^ (n % 8), zeros for tokens past the end
        const int lt = tid - 32 * DW_WARP_LOAD, n = lt >> 3, cc = lt & 7;
        constexpr int STEP = 32 * DW_LOAD_WARPS / 8;   // tokens a round
        static_assert(STEP % 8 == 0, "chunk positions of a thread's tokens");
        const uint32_t dst = sm0 + T::B + n * 128 + ((cc ^ (n & 7)) << 4);
        const size_t step = size_t(STEP) * p.K;
        bool alive = true;
        int ia = 0;                                    // stages so far, over all tiles
#pragma unroll 1
        for (int tile = blockIdx.x; tile < tiles && alive; tile += ONE ? tiles : int(gridDim.x)) {
            const int row0 = row_tile(tile) * DN_ROWS, n0 = token_tile(tile) * N, live = min(N, p.ntokens - n0);
            const int8_t* const src = p.q + size_t(n0) * p.K + 16 * cc;
#pragma unroll 1
            for (int i = 0; i < nst; ++i, ++ia) {
                const int b = ia & 1;
                if (!emptied(WB_B_EMPTY + b, ia >> 1, ERR_WAIT_PRODUCER)) { alive = false; break; }
                const bool two = 2 * i + 1 < ktot;
                const int8_t* at = src + size_t(n) * p.K + size_t(2 * i) * DN_GROUP;
#pragma unroll 4                               // more of them do not fit into 48 registers
                for (int k = 0; k < N / STEP; ++k, at += step) {
                    const bool on = n + STEP * k < live;
                    const int8_t* from = on ? at : src;
                    const uint32_t to = dst + b * 2 * T::B_GROUP + k * STEP * 128;
                    cp_async16(to, from, on);
                    if (two) cp_async16(to + T::B_GROUP, from + (on ? DN_GROUP : 0), on);
                }
                cp_async_arrive(BAR(WB_B_FULL + b));
                // the tile's part of Y into L2, wanted when the last group is folded
                if (i == 0)
                    for (int k = lt; k < live * 4; k += 32 * DW_LOAD_WARPS) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.Y + size_t(n0 + (k >> 2)) * p.rows + row0 + 32 * (k & 3)));
            }
        }
        cp_async_commit();
        cp_async_wait<0>();
    } else if (warp == DW_WARP_PRODUCER) {
        // ---- codes by bulk copy, one strip a lane
        int issued = 0;
        bool alive = true;
#pragma unroll 1
        for (int tile = blockIdx.x; tile < tiles && alive; tile += ONE ? tiles : int(gridDim.x)) {
            const uint8_t* strips = p.W + size_t(row_tile(tile) * (DN_ROWS / 16)) * strip_bytes;
#pragma unroll 1
            for (int i = 0; i < nst; ++i) {
                const int b = issued & 1;
                if (!emptied_warp(WB_RAW_EMPTY + b, issued >> 1, ERR_WAIT_PRODUCER)) { alive = false; break; }
                const uint32_t bytes = 2 * i + 1 < ktot ? 2 * DN_TILE_BYTES : DN_TILE_BYTES;
                if (lane == 0) ptx::mbar_arrive_expect_tx(BAR(WB_RAW_FULL + b), 8 * bytes);
                __syncwarp();
                if (lane < 8)
                    ptx::bulk_g2s(sm0 + T::RAW + b * 2 * T::RAW_GROUP + lane * 2 * DN_TILE_BYTES, strips + lane * strip_bytes + size_t(2 * i) * DN_TILE_BYTES, bytes, BAR(WB_RAW_FULL + b));
                ++issued;
            }
        }
        // copies still in flight must land before the shared memory is given back
        if (*abort_flag)
            for (int k = max(0, issued - DW_RAW); k < issued; ++k) {
                volatile int never = 0;
                ptx::mbar_wait(BAR(WB_RAW_FULL + (k & 1)), (k >> 1) & 1, &never);
            }
    } else {
        // ---- MMA issue (one elected lane issues, the warp stays together)
        const uint32_t hi = ptx::desc_hi(1024) | (2u << 29), idesc = idesc_i8_u8s8(DN_ROWS, N);
        const uint32_t a_lo = ptx::desc_lo(sm0 + T::A, 16), b_lo = ptx::desc_lo(sm0 + T::B, 16);
        bool alive = true;
        int ia = 0, ga = 0;                            // stages and groups so far, over all tiles
#pragma unroll 1
        for (int tile = blockIdx.x; tile < tiles && alive; tile += ONE ? tiles : int(gridDim.x)) {
#pragma unroll 1
            for (int i = 0; i < nst && alive; ++i, ++ia) {
                const int b = ia & 1, u = ia >> 1;
                if (!filled_warp(WB_B_FULL + b, u, ERR_WAIT_MMA) || !filled_warp(WB_A_FULL + b, u, ERR_WAIT_MMA)) { alive = false; break; }
                ptx::fence_proxy_async_smem();             // the activations, written by other threads' cp.async and seen through the barrier
#pragma unroll 1
                for (int e = 0; e < 2 && 2 * i + e < ktot; ++e, ++ga) {
                    const int slot = ga % DW_ACC;
                    if (!emptied_warp(WB_ACC_EMPTY + slot, ga / DW_ACC, ERR_WAIT_MMA)) { alive = false; break; }
                    ptx::tc_fence_after();
                    mma_i8_group_warp(tmem + slot * N, a_lo + (2 * b + e) * (T::A_GROUP / 16), b_lo + (2 * b + e) * (T::B_GROUP / 16), hi, idesc, BAR(WB_ACC_FULL + slot));
                }
                ptx::mma_commit_warp(BAR(WB_A_EMPTY + b));
                ptx::mma_commit_warp(BAR(WB_B_EMPTY + b));
            }
        }
        ptx::mma_commit_warp(BAR(WB_SPARE));           // every MMA issued must have retired before tensor memory is released
        volatile int never = 0;
        if (!ptx::mbar_wait(BAR(WB_SPARE), 0, &never)) errbits |= ERR_WAIT_TEARDOWN;
    }
    if (errbits) report_error(p, errbits);
    ptx::tc_fence_before();
    __syncthreads();
    if (warp == DW_WARP_MMA) ptx::tmem_dealloc(tmem, T::TMEM);
}

}  // namespace llattn
