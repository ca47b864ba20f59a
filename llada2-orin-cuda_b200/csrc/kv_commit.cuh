// Block-commit quantiser: a finished block's fp16 K/V -> one 4736-byte "4c/4" record per kv head.
// Replaces the reference's attn::kv_commit (engine/attn.cu:369-418) and must produce the same bytes:
//   K: per channel over the block's 32 tokens, V: per token over the 128 dims;
//   scale = half(max((max - min) / 15, 6.2e-5f)), min = half(min), code = clamp(rint((v - min) / scale), 0, 15),
//   all in IEEE fp32 with round-to-nearest-even; two codes per byte, even channel in the low nibble.
// One CTA per (kv head, block). The block's K and V slices sit in shared memory as fp16 tiles - loaded with 16-byte
// loads by kv_commit_kernel, or left there by the producer kernel that has just computed them (qkv_prepare.cuh) -, the
// record is assembled in shared memory and leaves as 16-byte stores.
#pragma once
#include <cuda_fp16.h>
#include "common.cuh"
#include "ptx.cuh"

namespace llattn {

constexpr int COMMIT_SHIM_THREADS = 128;        // the launch shape of the reference (attn_shim.cuh)

__device__ __forceinline__ void commit_meta(float mn, float mx, half& sh, half& mh) {
    sh = __float2half_rn(fmaxf(__fdiv_rn(__fsub_rn(mx, mn), 15.f), 6.2e-5f));
    mh = __float2half_rn(mn);
}
// clamp(rint((v - m0) / s), 0, 15) as a float, with the division rounded as IEEE says, r = 1 / s correctly rounded. The
// product with r is within 16 x 2^-22 of that quotient wherever the clamp lets the difference show, so only a product that
// lies this close to a tie (or is not finite) needs the division itself: about one value in a thousand. Rounding to an
// integer is the addition of 1.5 x 2^23 (larger products end at the clamp either way): the divisions and the conversion
// instructions, an eighth of the rate of an addition, were most of the kernel's time.
__device__ __forceinline__ float commit_code(float v, float m0, float s, float r) {
    const float x = __fsub_rn(v, m0), a = __fmul_rn(x, r);
    float n = __fsub_rn(__fadd_rn(a, 12582912.f), 12582912.f);
    if (!(fabsf(a - n) < 0.4995f)) n = rintf(__fdiv_rn(x, s));
    return fminf(fmaxf(n, 0.f), 15.f);
}
// Four codes, the first in the low nibble.
__device__ __forceinline__ uint32_t pack_codes(float c0, float c1, float c2, float c3) {
    return __float_as_uint(fmaf(c3, 4096.f, fmaf(c2, 256.f, fmaf(c1, 16.f, c0))) + 12582912.f) & 0xffffu;
}

constexpr int TILE_LD = D + 8;           // halves per tile row: rows 272 B apart, 16-byte aligned, no bank conflicts by column

// Shared memory of one (block, kv head) commit: the fp16 K and V slices, partial extrema of K, the assembled record.
struct CommitSmem {
    __align__(16) half Ks[BLK][TILE_LD];
    __align__(16) half Vs[BLK][TILE_LD];
    float kmin[4][D], kmax[4][D];
    __align__(16) uint8_t rec[REC_BYTES];
};

// The quantiser proper, from tiles already in shared memory (filled by 16-byte loads of fp16 K/V, or by the producer
// kernel that has just computed them) to the record at `dst`. NT = 128, 256 or 512 threads; the tiles must be complete (a
// __syncthreads before the call). What bounds it is the length of a thread's dependent chain (a commit is a few hundred
// CTAs at most), so a K channel is shared by NT / 128 threads, each with 32 / (NT / 128) tokens, and a warp's V tokens go
// through their shuffles together. fminf and fmaxf order -0 below +0 and pass NaN by whatever the order of the operands,
// so the extrema do not depend on the split.
// In a graph, 128 threads with a channel per thread and a division per value -> this: 1 block 9.5 -> 3.0 us, 64 blocks
// 10.2 -> 4.3, 2048 blocks 102 -> 68 (its bytes: 26).
template <int NT>
__device__ __forceinline__ void commit_tiles(CommitSmem& sm, uint8_t* __restrict__ dst, int tid) {
    constexpr int PARTS = NT / D, KT = BLK / PARTS, VT = BLK / (NT / 32);
    static_assert(PARTS >= 1 && PARTS <= 4 && KT % 8 == 0, "128, 256 or 512 threads");
    const int lane = tid & 31, warp = tid >> 5;
    // ---- K: a thread owns one channel of KT tokens
    const int c = tid & (D - 1), part = tid / D;
    half kv[KT];
    {
        float mn = INFINITY, mx = -INFINITY;
#pragma unroll
        for (int k = 0; k < KT; ++k) {
            kv[k] = sm.Ks[part * KT + k][c];
            const float v = __half2float(kv[k]);
            mn = fminf(mn, v); mx = fmaxf(mx, v);
        }
        sm.kmin[part][c] = mn; sm.kmax[part][c] = mx;
    }
    // ---- V: a warp takes tokens warp, warp + NT / 32, ...; a lane owns dims 4*lane .. 4*lane+3
    {
        float v[VT][4], mn[VT], mx[VT];
#pragma unroll
        for (int k = 0; k < VT; ++k) {
            const uint2 raw = *reinterpret_cast<const uint2*>(&sm.Vs[warp + k * (NT / 32)][lane * 4]);
            const half2 a = *reinterpret_cast<const half2*>(&raw.x), b = *reinterpret_cast<const half2*>(&raw.y);
            v[k][0] = __low2float(a); v[k][1] = __high2float(a); v[k][2] = __low2float(b); v[k][3] = __high2float(b);
            mn[k] = fminf(fminf(v[k][0], v[k][1]), fminf(v[k][2], v[k][3]));
            mx[k] = fmaxf(fmaxf(v[k][0], v[k][1]), fmaxf(v[k][2], v[k][3]));
        }
#pragma unroll
        for (int o = 16; o; o >>= 1)
#pragma unroll
            for (int k = 0; k < VT; ++k) {
                mn[k] = fminf(mn[k], __shfl_xor_sync(0xffffffffu, mn[k], o));
                mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], o));
            }
#pragma unroll
        for (int k = 0; k < VT; ++k) {
            const int tok = warp + k * (NT / 32);
            half sh, mh;
            commit_meta(mn[k], mx[k], sh, mh);
            const float s = __half2float(sh), m0 = __half2float(mh), r = __frcp_rn(s);
            const uint32_t packed = pack_codes(commit_code(v[k][0], m0, s, r), commit_code(v[k][1], m0, s, r),
                                               commit_code(v[k][2], m0, s, r), commit_code(v[k][3], m0, s, r));
            *reinterpret_cast<uint16_t*>(sm.rec + VOFF + tok * 64 + lane * 2) = uint16_t(packed);
            if (lane == 0) {
                reinterpret_cast<half*>(sm.rec + VOFF_META)[tok] = sh;
                reinterpret_cast<half*>(sm.rec + VOFF_META)[BLK + tok] = mh;
            }
        }
    }
    __syncthreads();
    {
        float mn = sm.kmin[0][c], mx = sm.kmax[0][c];
#pragma unroll
        for (int k = 1; k < PARTS; ++k) { mn = fminf(mn, sm.kmin[k][c]); mx = fmaxf(mx, sm.kmax[k][c]); }
        half sh, mh;
        commit_meta(mn, mx, sh, mh);
        const float s = __half2float(sh), m0 = __half2float(mh), r = __frcp_rn(s);
        // eight tokens' codes in a word; lanes of an even and an odd channel swap halves, each then has both nibbles of
        // four of the eight tokens' bytes
#pragma unroll
        for (int k0 = 0; k0 < KT; k0 += 8) {
            float code[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) code[k] = commit_code(__half2float(kv[k0 + k]), m0, s, r);
            const uint32_t w = pack_codes(code[0], code[1], code[2], code[3]) | pack_codes(code[4], code[5], code[6], code[7]) << 16;
            const uint32_t other = __shfl_xor_sync(0xffffffffu, w, 1);
            const uint32_t lo = (lane & 1) ? other >> 16 : w, hi = (lane & 1) ? w >> 16 : other;     // even channel, odd channel
            const int tok = part * KT + k0 + 4 * (lane & 1);
#pragma unroll
            for (int k = 0; k < 4; ++k) sm.rec[(tok + k) * 64 + (c >> 1)] = uint8_t(((lo >> (4 * k)) & 15u) | (((hi >> (4 * k)) & 15u) << 4));
        }
        if (part == 0) {
            reinterpret_cast<half*>(sm.rec + KOFF_META)[c] = sh;
            reinterpret_cast<half*>(sm.rec + KOFF_META)[D + c] = mh;
        }
    }
    __syncthreads();
    for (int i = tid; i < REC_BYTES / 16; i += NT)
        reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(sm.rec)[i];
}

// Kf, Vf: [nb][32 tok][4 heads][128] fp16. Record of (input block j, head h):
//   pages == nullptr: records + (h * max_blocks + blk + j) * 4736      (the reference's contiguous layer cache)
//   pages != nullptr: records + pages[j * 4 + h] * 4736                (record pool)
template <int NT>
__device__ __forceinline__ void kv_commit_body(const half* __restrict__ Kf, const half* __restrict__ Vf,
                                               uint8_t* __restrict__ records, const int32_t* __restrict__ pages,
                                               int max_blocks, int blk) {
    __shared__ CommitSmem sm;
    const int h = blockIdx.x, j = blockIdx.y, tid = threadIdx.x;
    const size_t in0 = size_t(j) * BLK * NKV * D + size_t(h) * D;
    const size_t ridx = pages ? size_t(pages[j * NKV + h]) : size_t(h) * max_blocks + blk + j;
    // ---- both slices into shared memory (32 tokens x 256 B each, 16-byte loads)
    constexpr int LOADS = BLK * D / 8 / NT;
    uint4 k4[LOADS], v4[LOADS];
#pragma unroll
    for (int i = 0; i < LOADS; ++i) {
        const size_t at = in0 + size_t((tid + NT * i) >> 4) * NKV * D + ((tid + NT * i) & 15) * 8;
        k4[i] = *reinterpret_cast<const uint4*>(Kf + at);
        v4[i] = *reinterpret_cast<const uint4*>(Vf + at);
    }
#pragma unroll
    for (int i = 0; i < LOADS; ++i) {
        const int tok = (tid + NT * i) >> 4, ch = (tid + NT * i) & 15;
        *reinterpret_cast<uint4*>(&sm.Ks[tok][ch * 8]) = k4[i];
        *reinterpret_cast<uint4*>(&sm.Vs[tok][ch * 8]) = v4[i];
    }
    __syncthreads();
    commit_tiles<NT>(sm, records + ridx * REC_BYTES, tid);
}

template <int NT>
__global__ void __launch_bounds__(NT)
kv_commit_kernel(const half* __restrict__ Kf, const half* __restrict__ Vf, uint8_t* __restrict__ records,
                 const int32_t* __restrict__ pages, int max_blocks, int blk) {
    ptx::grid_dependency_wait();               // nothing is read or written before the kernel ahead has completed
    kv_commit_body<NT>(Kf, Vf, records, pages, max_blocks, blk);
}

}  // namespace llattn
