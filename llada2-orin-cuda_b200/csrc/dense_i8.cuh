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
// Both kernels use mma.sync m16n8k32 (u8 x s8 -> s32), whose fragments these layouts are: a lane's eight code words ARE its
// A fragments (one nibble mask per register) and a token's B fragments are 32 contiguous bytes per lane, so operands go
// from memory to the tensor core without being unpacked into shared memory, and the integers come out in registers,
// where the fold into fp32 needs them. What the path costs is that fold, 16 float steps per output which cannot be
// reordered, not the products: the tcgen05 form (unpack to shared memory, proxy fence, MMA, commit, tensor-memory load)
// took 1.2 us for every group at any number of tokens, a chain longer than the group's arithmetic.
//   dense_strip_kernel  a decode step's few tokens: a CTA takes ONE strip and one warp per 128-group works on it; the
//                       integers of all groups exist at once, only the multiply-adds run in group order.
//   dense_tile_kernel   many tokens: 128 rows x 16, 32 or 64 tokens per CTA.
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
};

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

}  // namespace llattn
