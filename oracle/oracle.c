/*
 * CPU oracle for the block-diffusion attention path over the "4c/4" int4 KV cache.
 *
 * TEST INFRASTRUCTURE ONLY. The CUDA path is compared with this file; nothing that ships may
 * call it. It restates, in plain C, the arithmetic of the reference engine:
 *   - record layout                         engine/attn.cu:3-7,22-25
 *   - block-commit quantiser (kv_commit)    engine/attn.cu:369-418
 *   - record dequantisation                 engine/attn.cu:95-122 (fp16 fused multiply-add form)
 *                                           engine/tests/test_attn.cu:52-58 (exact code*scale+min form)
 *   - attention over [cache | fresh block]  engine/tests/test_attn.cu:75-95 (fp64 softmax, scale 1/sqrt(128))
 *   - prefill visibility (block j sees nblocks + j records and its own fresh block)
 *                                           engine/attn.cu:150-158, engine/engine.cu:591-598
 *   - int8 activation epilogue              engine/attn.cu:308-312,346-357
 *   - simulated quantiser in fp32           quant/s06_arbitrate.py:78-89 (fake_quant), applied per channel over
 *                                           32 tokens for K and per token for V as quant/student_case.py:63-66
 * Parity pinning: the packer/dequantiser pair is checked bit for bit against outputs of the reference's own
 * fake_quant (fixtures under tests/golden, generated by importing the reference in the build container).
 *
 * Build: gcc -O2 -fopenmp -ffp-contract=off -shared -fPIC oracle.c -o liboracle.so -lm
 * (-ffp-contract=off keeps q*s + mn as two roundings, as torch computes it.)
 */
#include <math.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>
#ifdef _OPENMP
#include <omp.h>
#endif

enum { D = 128, BLK = 32, NKV = 4, NQH = 16, GQA = 4 };
enum { REC_BYTES = 4736, KOFF_META = 2048, VOFF = 2560, VOFF_META = 4608 };

/* ---------------------------------------------------------------- fp16 <-> fp32/fp64, IEEE, round-half-even */

static inline float h2f(uint16_t h) {
    const uint32_t s = (uint32_t)(h >> 15) << 31, e = (h >> 10) & 31, m = h & 1023;
    uint32_t u;
    if (e == 0) {
        if (m == 0) u = s;
        else {                                   /* subnormal: value = m * 2^-24 */
            const float v = (float)m * 5.9604644775390625e-08f;
            memcpy(&u, &v, 4);
            u |= s;
        }
    } else if (e == 31) u = s | 0x7f800000u | (m << 13);
    else u = s | ((e + 112) << 23) | (m << 13);
    float f;
    memcpy(&f, &u, 4);
    return f;
}

/* double -> fp16 with one rounding (round to nearest, ties to even). */
static inline uint16_t d2h(double x) {
    uint64_t u;
    memcpy(&u, &x, 8);
    const uint16_t s = (uint16_t)((u >> 63) << 15);
    const double a = fabs(x);
    if (isnan(x)) return (uint16_t)(s | 0x7e00);
    if (a >= 65520.0) return (uint16_t)(s | 0x7c00);          /* rounds to inf */
    if (a < 6.103515625e-05) {                                 /* subnormal or zero: quantum 2^-24 */
        const double q = nearbyint(a * 16777216.0);            /* RNE under the default rounding mode */
        return (uint16_t)(s | (uint16_t)q);                    /* q == 1024 lands on the smallest normal */
    }
    int ex;
    const double fr = frexp(a, &ex);                           /* a = fr * 2^ex, fr in [0.5,1) */
    double m = nearbyint(fr * 2048.0);                         /* 11 significant bits */
    if (m == 2048.0) { m = 1024.0; ex += 1; }
    const int e = ex - 1 + 15;
    return (uint16_t)(s | (uint16_t)(e << 10) | ((uint16_t)m & 1023));
}
static inline uint16_t f2h(float f) { return d2h((double)f); }  /* float -> double is exact */

uint16_t orc_f2h(float f) { return f2h(f); }
float orc_h2f(uint16_t h) { return h2f(h); }

/* ---------------------------------------------------------------- the packer (engine/attn.cu:369-418) */

/* fminf/fmaxf as the GPU evaluates them: -0 orders below +0, whatever the argument order (checked on B200: a
 * group whose smallest values are +0 and -0 stores 0x8000 as its min). Inputs carry no NaN. */
static inline float minf_(float a, float b) { return (b < a || (b == a && signbit(b))) ? b : a; }
static inline float maxf_(float a, float b) { return (b > a || (b == a && !signbit(b))) ? b : a; }
static inline int clamp15(float q) {                          /* __float2int_rn then clamp to [0,15] */
    const long r = lrintf(q);
    return r < 0 ? 0 : (r > 15 ? 15 : (int)r);
}

/* scale/min of one group from its fp32 min and max: fp16 scale with the 6.2e-5 floor, fp16 min. */
static inline void group_meta(float mn, float mx, uint16_t* sh, uint16_t* mh) {
    *sh = f2h(maxf_((mx - mn) / 15.0f, 6.2e-5f));
    *mh = f2h(mn);
}

/* One record: K/V block given as [32 tok][row_stride halves] slices for one kv head (128 halves each row). */
static void pack_record(const uint16_t* K, const uint16_t* V, size_t row_stride, uint8_t* rec) {
    uint8_t kq[BLK][D], vq[BLK][D];
    uint16_t* kmeta = (uint16_t*)(rec + KOFF_META);
    uint16_t* vmeta = (uint16_t*)(rec + VOFF_META);
    for (int c = 0; c < D; ++c) {                              /* K: per channel over the 32 tokens */
        float mn = INFINITY, mx = -INFINITY;
        for (int t = 0; t < BLK; ++t) {
            const float v = h2f(K[t * row_stride + c]);
            mn = minf_(mn, v); mx = maxf_(mx, v);
        }
        uint16_t sh, mh;
        group_meta(mn, mx, &sh, &mh);
        const float s = h2f(sh), m0 = h2f(mh);
        for (int t = 0; t < BLK; ++t) kq[t][c] = (uint8_t)clamp15((h2f(K[t * row_stride + c]) - m0) / s);
        kmeta[c] = sh; kmeta[D + c] = mh;
    }
    for (int t = 0; t < BLK; ++t) {                            /* V: per token over the 128 dims */
        float mn = INFINITY, mx = -INFINITY;
        for (int c = 0; c < D; ++c) {
            const float v = h2f(V[t * row_stride + c]);
            mn = minf_(mn, v); mx = maxf_(mx, v);
        }
        uint16_t sh, mh;
        group_meta(mn, mx, &sh, &mh);
        const float s = h2f(sh), m0 = h2f(mh);
        for (int c = 0; c < D; ++c) vq[t][c] = (uint8_t)clamp15((h2f(V[t * row_stride + c]) - m0) / s);
        vmeta[t] = sh; vmeta[BLK + t] = mh;
    }
    for (int t = 0; t < BLK; ++t)                              /* byte = channel 2i | channel 2i+1 << 4 */
        for (int i = 0; i < D / 2; ++i) {
            rec[t * 64 + i] = (uint8_t)(kq[t][2 * i] | (kq[t][2 * i + 1] << 4));
            rec[VOFF + t * 64 + i] = (uint8_t)(vq[t][2 * i] | (vq[t][2 * i + 1] << 4));
        }
}

/* Kf, Vf: [nb][32][4][128] fp16. cache: [4][max_blocks][4736]. Block j of the input becomes record blk + j. */
void orc_kv_commit(const uint16_t* Kf, const uint16_t* Vf, uint8_t* cache, int max_blocks, int blk, int nb) {
#pragma omp parallel for collapse(2) schedule(static)
    for (int j = 0; j < nb; ++j)
        for (int h = 0; h < NKV; ++h) {
            const size_t in = (size_t)j * BLK * NKV * D + (size_t)h * D;
            pack_record(Kf + in, Vf + in, (size_t)NKV * D, cache + ((size_t)h * max_blocks + blk + j) * REC_BYTES);
        }
}

/* ---------------------------------------------------------------- dequantisation of one record
 * mode 0: exact code*scale + min in double                      (engine/tests/test_attn.cu:57-58)
 * mode 1: one fused multiply-add rounded to fp16                (engine/attn.cu:112-115, __hfma2)
 * mode 2: fp32 q*s + mn, two roundings                          (quant/s06_arbitrate.py:89)
 * K, V: [32][128] doubles. */
void orc_dequant_record(const uint8_t* rec, int mode, double* K, double* V) {
    const uint16_t* km = (const uint16_t*)(rec + KOFF_META);
    const uint16_t* vm = (const uint16_t*)(rec + VOFF_META);
    for (int t = 0; t < BLK; ++t)
        for (int c = 0; c < D; ++c) {
            const int kc = (rec[t * 64 + c / 2] >> (4 * (c & 1))) & 15;
            const int vc = (rec[VOFF + t * 64 + c / 2] >> (4 * (c & 1))) & 15;
            const float ks = h2f(km[c]), kmin = h2f(km[D + c]), vs = h2f(vm[t]), vmin = h2f(vm[BLK + t]);
            double k = (double)kc * ks + kmin, v = (double)vc * vs + vmin;   /* exact in double */
            if (mode == 1) { k = h2f(d2h(k)); v = h2f(d2h(v)); }
            else if (mode == 2) {
                const float kp = (float)kc * ks, vp = (float)vc * vs;
                k = (double)(kp + kmin); v = (double)(vp + vmin);
            }
            K[t * D + c] = k; V[t * D + c] = v;
        }
}

/* ---------------------------------------------------------------- attention (engine/tests/test_attn.cu:75-95)
 * One sequence. Q [nb][32][16][128], Kf/Vf [nb][32][4][128] fp16; cache [4][max_blocks][4736] or, when pages is
 * non-null, a record pool addressed as pool + pages[h * max_blocks + b] * 4736. Query block j attends records
 * 0 .. nblocks + j - 1 and its own fresh block, softmax over all of them, scale = 1/sqrt(128).
 * dq_mode selects the record dequantisation (see orc_dequant_record).
 * acc_f32 != 0: scores, softmax and PV accumulate in fp32 (the simulated-quantisation flavour); else fp64.
 * O: [nb*32][16][128] float, LSE: [nb*32][16] float (natural log of the softmax denominator, max included). */
void orc_attention(const uint16_t* Q, const uint16_t* Kf, const uint16_t* Vf, const uint8_t* cache,
                   const int32_t* pages, int max_blocks, int nblocks, int nb, int dq_mode, int acc_f32,
                   float* O, float* LSE) {
    const int nrec_max = nblocks + nb - 1;
    const size_t ctx_max = (size_t)(nrec_max + 1) * BLK;
    /* dequantise every record once per head */
    double* Kd = (double*)malloc(sizeof(double) * NKV * (size_t)(nrec_max > 0 ? nrec_max : 1) * BLK * D);
    double* Vd = (double*)malloc(sizeof(double) * NKV * (size_t)(nrec_max > 0 ? nrec_max : 1) * BLK * D);
#pragma omp parallel for collapse(2) schedule(static)
    for (int h = 0; h < NKV; ++h)
        for (int b = 0; b < nrec_max; ++b) {
            const size_t ridx = pages ? (size_t)pages[(size_t)h * max_blocks + b] : (size_t)h * max_blocks + b;
            const size_t o = ((size_t)h * nrec_max + b) * BLK * D;
            orc_dequant_record(cache + ridx * REC_BYTES, dq_mode, Kd + o, Vd + o);
        }
    const double scale = 1.0 / sqrt((double)D);
#pragma omp parallel
    {
        double* sc = (double*)malloc(sizeof(double) * ctx_max);
        double* kf = (double*)malloc(sizeof(double) * BLK * D);
        double* vf = (double*)malloc(sizeof(double) * BLK * D);
        double q[D];
#pragma omp for collapse(2) schedule(dynamic, 1)
        for (int j = 0; j < nb; ++j)
            for (int qh = 0; qh < NQH; ++qh) {
                const int h = qh / GQA, nrec = nblocks + j, ctx = (nrec + 1) * BLK;
                for (int t = 0; t < BLK; ++t)
                    for (int c = 0; c < D; ++c) {
                        const size_t i = ((size_t)j * BLK + t) * NKV * D + (size_t)h * D + c;
                        kf[t * D + c] = h2f(Kf[i]); vf[t * D + c] = h2f(Vf[i]);
                    }
                const double* Kh = Kd + (size_t)h * nrec_max * BLK * D;
                const double* Vh = Vd + (size_t)h * nrec_max * BLK * D;
                for (int t = 0; t < BLK; ++t) {
                    const size_t row = (size_t)j * BLK + t;
                    for (int c = 0; c < D; ++c) q[c] = h2f(Q[(row * NQH + qh) * D + c]);
                    float* out = O + (row * NQH + qh) * D;
                    if (!acc_f32) {
                        double mx = -1e300;
                        for (int k = 0; k < ctx; ++k) {
                            const double* kr = k < nrec * BLK ? Kh + (size_t)k * D : kf + (size_t)(k - nrec * BLK) * D;
                            double s = 0;
                            for (int c = 0; c < D; ++c) s += q[c] * kr[c];
                            sc[k] = s * scale;
                            if (sc[k] > mx) mx = sc[k];
                        }
                        double l = 0, acc[D];
                        for (int c = 0; c < D; ++c) acc[c] = 0;
                        for (int k = 0; k < ctx; ++k) {
                            const double p = exp(sc[k] - mx);
                            l += p;
                            const double* vr = k < nrec * BLK ? Vh + (size_t)k * D : vf + (size_t)(k - nrec * BLK) * D;
                            for (int c = 0; c < D; ++c) acc[c] += p * vr[c];
                        }
                        for (int c = 0; c < D; ++c) out[c] = (float)(acc[c] / l);
                        LSE[row * NQH + qh] = (float)(mx + log(l));
                    } else {
                        float mx = -INFINITY;
                        float* scf = (float*)sc;
                        const float scalef = (float)scale;
                        for (int k = 0; k < ctx; ++k) {
                            const double* kr = k < nrec * BLK ? Kh + (size_t)k * D : kf + (size_t)(k - nrec * BLK) * D;
                            float s = 0.f;
                            for (int c = 0; c < D; ++c) s += (float)q[c] * (float)kr[c];
                            scf[k] = s * scalef;
                            if (scf[k] > mx) mx = scf[k];
                        }
                        float l = 0.f, acc[D];
                        for (int c = 0; c < D; ++c) acc[c] = 0.f;
                        for (int k = 0; k < ctx; ++k) {
                            const float p = expf(scf[k] - mx);
                            l += p;
                            const double* vr = k < nrec * BLK ? Vh + (size_t)k * D : vf + (size_t)(k - nrec * BLK) * D;
                            for (int c = 0; c < D; ++c) acc[c] += p * (float)vr[c];
                        }
                        for (int c = 0; c < D; ++c) out[c] = acc[c] / l;
                        LSE[row * NQH + qh] = mx + logf(l);
                    }
                }
            }
        free(sc); free(kf); free(vf);
    }
    free(Kd); free(Vd);
}

/* ---------------------------------------------------------------- int8 activation epilogue (engine/attn.cu:308-312,346-357)
 * O: [rows][16][128] float -> q8 [rows][2048] in fragment order, s8 [rows][16], sum8 [rows][16]. */
static inline int frag_pos(int c) {
    const int base = c & ~127, r = c & 127;
    return base + 32 * ((r >> 2) & 3) + 8 * (r >> 5) + 4 * ((r >> 4) & 1) + (r & 3);
}
int orc_frag_pos(int c) { return frag_pos(c); }

void orc_act_q8(const float* O, int rows, int8_t* q8, float* s8, int32_t* sum8) {
    for (int r = 0; r < rows; ++r)
        for (int h = 0; h < NQH; ++h) {
            const float* v = O + ((size_t)r * NQH + h) * D;
            float m = 0.f;
            for (int c = 0; c < D; ++c) m = maxf_(m, fabsf(v[c]));
            const float sc = maxf_(m / 127.0f, 1e-30f);
            int sm = 0;
            for (int c = 0; c < D; ++c) {
                long q = lrintf(v[c] / sc);
                q = q < -127 ? -127 : (q > 127 ? 127 : q);
                q8[(size_t)r * 2048 + frag_pos(h * D + c)] = (int8_t)q;
                sm += (int)q;
            }
            s8[r * NQH + h] = sc; sum8[r * NQH + h] = sm;
        }
}

/* ---------------------------------------------------------------- simulated quantiser (quant/s06_arbitrate.py:78-89)
 * x: [ngroups][group] float in, dequantised q*s + mn out (fp32, two roundings). bits = 4. */
void orc_fake_quant(const float* x, float* y, size_t ngroups, int group) {
#pragma omp parallel for schedule(static)
    for (size_t g = 0; g < ngroups; ++g) {
        const float* xi = x + g * group;
        float mn = INFINITY, mx = -INFINITY;
        for (int i = 0; i < group; ++i) { mn = minf_(mn, xi[i]); mx = maxf_(mx, xi[i]); }
        const float s = h2f(f2h(maxf_((mx - mn) / 15.0f, 6.2e-5f))), m0 = h2f(f2h(mn));
        for (int i = 0; i < group; ++i) {
            float q = nearbyintf((xi[i] - m0) / s);
            q = q < 0.f ? 0.f : (q > 15.f ? 15.f : q);
            const float p = q * s;
            y[g * group + i] = p + m0;
        }
    }
}

int orc_num_threads(void) {
#ifdef _OPENMP
    return omp_get_max_threads();
#else
    return 1;
#endif
}

/* ---------------------------------------------------------------- producer of the attention inputs (engine/ops.cu:429-453)
 * qkv [T][3072] fp32 (16 q heads, 4 k heads, 4 v heads of 128) -> q [T][16][128], k, v [T][4][128] fp16.
 * Per q/k head: RMSNorm (mean of squares over 128 dims + eps, weights gq / gk), then RoPE on dims 0..63 with the
 * rotate-half pairing (d, d + 32), angle pos[t] * inv_freq[d], cos/sin rounded to bf16; dims 64..127 only normalised;
 * v converted. Evaluated in double with the same roundings to bf16 (cos/sin) and fp16 (outputs); n = x*r*g is kept in
 * double, so the GPU's fp32 arithmetic may differ from this by an fp16 ulp, and by one bf16 ulp of cos/sin where
 * sincosf's last-bit error crosses a bf16 rounding boundary. */
static double bf16_round(double x) {
    float f = (float)x;
    uint32_t u;
    memcpy(&u, &f, 4);
    const uint32_t lsb = (u >> 16) & 1u;
    u += 0x7fffu + lsb;                      /* round to nearest even on the upper 16 bits */
    u &= 0xffff0000u;
    memcpy(&f, &u, 4);
    return (double)f;
}

void orc_qk_norm_rope(const float* qkv, const int32_t* pos, const float* gq, const float* gk, float eps,
                      const float* inv_freq, uint16_t* q, uint16_t* k, uint16_t* v, int T) {
#pragma omp parallel for schedule(static)
    for (int t = 0; t < T; ++t)
        for (int hd = 0; hd < 24; ++hd) {
            const float* x = qkv + (size_t)t * 3072 + hd * 128;
            if (hd >= 20) {
                for (int d = 0; d < D; ++d) v[((size_t)t * NKV + (hd - 20)) * D + d] = f2h(x[d]);
                continue;
            }
            double ss = 0;
            for (int d = 0; d < D; ++d) ss += (double)x[d] * x[d];
            const double r = 1.0 / sqrt(ss / 128.0 + (double)eps);
            const float* g = hd < 16 ? gq : gk;
            uint16_t* dst = hd < 16 ? q + ((size_t)t * NQH + hd) * D : k + ((size_t)t * NKV + (hd - 16)) * D;
            for (int l = 0; l < 32; ++l) {
                const double n0 = x[l] * r * g[l], n1 = x[l + 32] * r * g[l + 32];
                const float ang = (float)pos[t] * inv_freq[l];           /* fp32 product, as the kernel forms the angle */
                const double cs = bf16_round(cos((double)ang)), sn = bf16_round(sin((double)ang));
                dst[l] = d2h(n0 * cs - n1 * sn);
                dst[l + 32] = d2h(n1 * cs + n0 * sn);
                dst[l + 64] = d2h(x[l + 64] * r * g[l + 64]);
                dst[l + 96] = d2h(x[l + 96] * r * g[l + 96]);
            }
        }
}

/* ---- dense W4.A8 projection with residual add: restates what the engine's attention-output projection computes
 * (engine/engine.cu:434 -> moe8::gemm MODE 2, engine/moe_i8.cu:295-400, single K split): per output the exact integer
 * group products (tile code layout engine/moe_i8.cu:127-160, activations in fragment order engine/moe_i8.cu:55-60),
 * then one fp32 product of the two scales and one fused multiply-add per 128-group in ascending order
 * (engine/moe_i8.cu:374-380), then one add into Y (engine/moe_i8.cu:236-244).
 * W: rows / 16 strips, each K/128 code tiles of 1024 bytes followed by K/128 metas of 48 bytes (engine/moe_i8.cu:34-41). */
void orc_dense_w4a8(const uint8_t* W, const int8_t* q, const float* s, const int32_t* sum, float* Y, int ntokens, int rows, int K) {
    const int ktot = K / 128;
    const size_t strip_bytes = (size_t)ktot * (1024 + 48);
#pragma omp parallel for schedule(static)
    for (int r = 0; r < rows; ++r) {
        const int strip = r >> 4, rr = r & 15, g = rr & 7, hi = rr >> 3;
        const uint8_t* sp = W + (size_t)strip * strip_bytes;
        for (int n = 0; n < ntokens; ++n) {
            float c = 0.f;
            for (int kt = 0; kt < ktot; ++kt) {
                const uint8_t* tile = sp + (size_t)kt * 1024;
                const uint8_t* meta = sp + (size_t)ktot * 1024 + (size_t)kt * 48;
                uint16_t hs;
                memcpy(&hs, meta + 4 * g + 2 * hi, 2);
                const float sw = h2f(hs);
                const int z = meta[32 + 2 * g + hi];
                const int8_t* x = q + (size_t)n * K + (size_t)kt * 128;
                int P = 0;
                for (int t = 0; t < 4; ++t)
                    for (int w = 0; w < 8; ++w)
                        for (int e = 0; e < 4; ++e) {
                            const uint8_t byte = tile[(w < 4 ? 0 : 512) + 16 * (4 * g + t) + 4 * (w & 3) + e];
                            const int code = hi ? byte >> 4 : byte & 15;
                            const int j = w >> 1, h = w & 1;                 /* logical k = 32 j + 16 h + 4 t + e */
                            P += code * (int)x[32 * t + 8 * j + 4 * h + e];   /* its fragment position */
                        }
                const int v = P - z * sum[(size_t)n * ktot + kt];
                const float ss = sw * s[(size_t)n * ktot + kt];
                c = fmaf(ss, (float)v, c);
            }
            Y[(size_t)n * rows + r] += c;
        }
    }
}
