// Producer of the attention inputs, fused with the block commit for prefill.
//
// Stands in for the reference's ops::qk_norm_rope (engine/ops.cu:429-453): per head RMSNorm of q and k with a learned
// gain, rotary embedding on the first 64 dims of each head (rotate-half pairs (d, d + 32), cos/sin rounded to bf16 as
// the model computes them), v converted; fp32 qkv [T][3072] (16 q heads, 4 k heads, 4 v heads of 128) in, fp16 Q [T][16][128]
// and fresh K, V [T][4][128] out. In a prefill pass the reference then runs attn::kv_commit on those fp16 K/V
// (engine/engine.cu:589-591), reading them back from memory; here the CTA that produces a 32-token block of one kv
// head keeps the fp16 K and V it has just rounded in shared memory and quantises the block's record from there
// (kv_commit.cuh), so a prefill block goes from fp32 qkv to its 4736-byte record in one pass: 12,288 B read and
// 6,144 + 592 B written per token, against 14,336 read and the same written by the two-kernel sequence.
//
// A warp takes the four heads of one group for one token: sixteen loads in flight, one sine and cosine for all of them.
// Groups 0-3 are q heads, 4 the k heads, 5 the v heads; grid (blocks of 32 tokens, 24): group y / 4, tokens 8 (y % 4) ..,
// 8 warps a CTA. With the commit, K and V of a (block, kv head) stay with one CTA: grid (blocks, 4 + 16), y < 4 kv head y, a warp per four
// tokens, then the q groups as above. These four have the longest way and come first in the grid (52 blocks 8.0 -> 7.0 us in a graph,
// 16 blocks 6.1 -> 5.2). For few blocks CTAs have 512 threads (grid (blocks, 4 + 8), a warp per two tokens of K and V: one block 4.6 ->
// 3.7 us, 16 5.2 -> 4.5, 52 6.9 -> 6.7, 64 7.8 -> 7.7, 74 8.4 -> 8.6): up to 65 on 148 SMs, with 1.75 of the longer CTAs an SM.
// Bound by latency in a decode step: the former split, 8 CTAs per block whose warps walked 16 rows one after the
// other, took 7.8 us for one block in a graph; now 1.6 (with the commit 9.5 -> 3.7). HBM-bound from a few thousand tokens
// on: 8192 tokens 38.9 -> 24.6 us = 6.1 TB/s.
// Lane l holds dims l, l+32, l+64, l+96 of a row: the rotate-half partners
// then share a lane and every global access of a warp is one contiguous segment. The float operations and their order
// are the reference kernel's (sum of squares folded lane-wise then by a xor butterfly, rsqrtf, x*r*g, sincosf, one
// fused multiply-add per rotated output), which is what makes the outputs bit-identical to it.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include "common.cuh"
#include "ptx.cuh"
#include "kv_commit.cuh"

namespace llattn {

constexpr int PREP_THREADS = 256, PREP_FEW_THREADS = 512;      // with the commit, few blocks: the latter
__host__ __device__ constexpr int prep_parts(int threads) { return BLK / (threads / 32); }      // CTAs that share a group's tokens of a block

struct PrepArgs {
    const float* qkv;        // [T][3072]
    const int* pos;          // [T]
    const float* gq;         // [128]
    const float* gk;         // [128]
    const float* inv_freq;   // [32]
    float eps;
    half* q;                 // [T][16][128]
    half* k;                 // [T][4][128]
    half* v;                 // [T][4][128]
    int T;
    // commit of the blocks this launch produces (records == nullptr: none). Block j of the launch, head h:
    // pages ? records + pages[j * 4 + h] * 4736 : records + (h * max_blocks + blk + j) * 4736
    uint8_t* records;
    const int32_t* pages;
    int max_blocks, blk;
};

// One head row of a token: the four values a lane holds, normalised and rotated in place.
__device__ __forceinline__ void norm_rope_lane(float (&x)[4], const float* __restrict__ gain, int lane, float eps, float cs, float sn) {
    float ss = x[0] * x[0] + x[1] * x[1] + x[2] * x[2] + x[3] * x[3];
#pragma unroll
    for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float r = rsqrtf(ss / 128.f + eps);
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = x[i] * r * gain[lane + 32 * i];
    // written out: the first product of each pair goes into the fused multiply-add, the second is rounded on its own.
    // That is what the compiler makes of the reference's `n0 * cs - n1 * sn` and `n1 * cs + n0 * sn`, and the other
    // choice differs from it in the last fp16 bit of about one output in 20,000.
    const float lo = __fmaf_rn(x[0], cs, -__fmul_rn(x[1], sn));
    const float hi = __fmaf_rn(x[1], cs, __fmul_rn(x[0], sn));
    x[0] = lo; x[1] = hi;
}

__device__ __forceinline__ void rope_angle(const PrepArgs& a, int t, float freq, float& cs, float& sn) {
    sincosf(float(a.pos[t]) * freq, &sn, &cs);
    cs = __bfloat162float(__float2bfloat16(cs));
    sn = __bfloat162float(__float2bfloat16(sn));
}

template <bool COMMIT, int NT>
__global__ void __launch_bounds__(NT) qkv_prepare_kernel(const PrepArgs a) {
    ptx::grid_dependency_wait();               // nothing is read or written before the kernel ahead has completed
    const int jb = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t0 = jb * BLK;
    const float freq = a.inv_freq[lane];
    if (!COMMIT || blockIdx.y >= NKV) {
        // ---- four heads of one token
        const int part = int(blockIdx.y) - (COMMIT ? NKV : 0), grp = part / prep_parts(NT), t = t0 + NT / 32 * (part % prep_parts(NT)) + warp;
        if (t >= a.T) return;
        const float* src = a.qkv + size_t(t) * 3072 + 4 * grp * D + lane;
        float x[4][4];
#pragma unroll
        for (int h = 0; h < 4; ++h)
#pragma unroll
            for (int c = 0; c < 4; ++c) x[h][c] = src[h * D + 32 * c];
        if (grp < 5) {
            const float* gain = grp < 4 ? a.gq : a.gk;
            float cs, sn;
            rope_angle(a, t, freq, cs, sn);
#pragma unroll
            for (int h = 0; h < 4; ++h) norm_rope_lane(x[h], gain, lane, a.eps, cs, sn);
        }
        half* dst = (grp < 4 ? a.q + (size_t(t) * NQH + 4 * grp) * D : (grp == 4 ? a.k : a.v) + size_t(t) * NKV * D) + lane;
#pragma unroll
        for (int h = 0; h < 4; ++h)
#pragma unroll
            for (int c = 0; c < 4; ++c) dst[h * D + 32 * c] = __float2half(x[h][c]);
        return;
    }
    if constexpr (COMMIT) {
        // ---- kv head h: the block's K (normalised, rotated) and V (converted) as fp16 tiles in shared memory. Whole blocks.
        __shared__ CommitSmem sm;
        const int h = blockIdx.y;
        constexpr int TOKS = BLK / (NT / 32);
        float xk[TOKS][4], xv[TOKS][4];
#pragma unroll
        for (int k = 0; k < TOKS; ++k) {
            const float* ks = a.qkv + size_t(t0 + TOKS * warp + k) * 3072 + (NQH + h) * D + lane;
#pragma unroll
            for (int c = 0; c < 4; ++c) { xk[k][c] = ks[32 * c]; xv[k][c] = ks[NKV * D + 32 * c]; }
        }
#pragma unroll
        for (int k = 0; k < TOKS; ++k) {
            const int tok = TOKS * warp + k;
            float cs, sn;
            rope_angle(a, t0 + tok, freq, cs, sn);
            norm_rope_lane(xk[k], a.gk, lane, a.eps, cs, sn);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                sm.Ks[tok][lane + 32 * c] = __float2half(xk[k][c]);
                sm.Vs[tok][lane + 32 * c] = __float2half(xv[k][c]);
            }
        }
        __syncthreads();
        // ---- fp16 K and V of the block to global memory, 16 bytes per thread and store
        for (int i = threadIdx.x; i < BLK * 16; i += NT) {
            const int tok = i >> 4, ch = i & 15;
            const size_t at = (size_t(t0 + tok) * NKV + h) * D + ch * 8;
            *reinterpret_cast<uint4*>(a.k + at) = *reinterpret_cast<const uint4*>(&sm.Ks[tok][ch * 8]);
            *reinterpret_cast<uint4*>(a.v + at) = *reinterpret_cast<const uint4*>(&sm.Vs[tok][ch * 8]);
        }
        const size_t ridx = a.pages ? size_t(a.pages[jb * NKV + h]) : size_t(h) * a.max_blocks + a.blk + jb;
        commit_tiles<NT>(sm, a.records + ridx * REC_BYTES, threadIdx.x);
    }
}

}  // namespace llattn
