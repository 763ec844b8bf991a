// Causal prompt attention on the tensor cores with fp32-grade accuracy: S = Q K^T and O = P V as bf16 MMAs
// (mma.sync.m16n8k16, fp32 accumulate) on operands split three ways, x = hi + mid + lo with each part a bf16
// (8 + 8 + 8 mantissa bits = the 24 of fp32).  A product keeps the six terms hi*hi, hi*mid, mid*hi, hi*lo, lo*hi,
// mid*mid; what is dropped is below 2^-24 of the product, so scores and outputs carry fp32 rounding only
// (ScaledDotProductFlash*'s arithmetic up to summation order, AttentionKernels.cs:220-475).  Six MMAs of 2048
// multiply-adds replace 12 288 fp32 FMAs, i.e. 384 warp instructions: the CUDA-core kernel this replaces spent its
// time waiting on shared-memory operands of those FMAs.
//
// One CTA = 64 consecutive query rows of HPC (1 or 2) query heads that share a KV head, four warps per head, 16 rows
// per warp.  K and V go through shared memory in tiles of 32 keys, split into their three bf16 planes ONCE per CTA
// while they are staged (rows padded to an odd multiple of 16 bytes: every ldmatrix is conflict free); Q is split
// the same way once per CTA.  The score tile's accumulator layout is the A-operand layout of the next MMA for
// 16-bit types, so P goes from registers to registers.  Online softmax per row as in the scalar kernel.
// sm_100a runs mma.sync on its legacy tensor path.  smc_attention_tc.cu is the tcgen05 form, with the same bits; this kernel stays for calls of
// one to a few key tiles, outputs off 16 bytes, one head per CTA (an option) and calls that the other's planes do not reach (a very long cache, a full device).
#include <cuda_bf16.h>

#include "smc_common.cuh"

#include <type_traits>

namespace {

constexpr int QROWS = 64, KT = 32;

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4])
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm4t(uint32_t addr, uint32_t (&r)[4])
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
// x = hi + mid + lo, each a bf16 (round to nearest; the remainders are exact in fp32)
__device__ __forceinline__ void split3(float x, __nv_bfloat16 &hi, __nv_bfloat16 &mid, __nv_bfloat16 &lo)
{
    hi = __float2bfloat16_rn(x);
    const float r1 = x - __bfloat162float(hi);
    mid = __float2bfloat16_rn(r1);
    lo = __float2bfloat16_rn(r1 - __bfloat162float(mid));
}
__device__ __forceinline__ uint32_t pack2(__nv_bfloat16 a, __nv_bfloat16 b)
{
    return (uint32_t)__bfloat16_as_ushort(a) | ((uint32_t)__bfloat16_as_ushort(b) << 16);
}
// the six kept terms of (a_hi + a_mid + a_lo) * (b_hi + b_mid + b_lo), smallest first
__device__ __forceinline__ void mma6(float (&c)[4], const uint32_t (&ah)[4], const uint32_t (&am)[4], const uint32_t (&al)[4],
                                     const uint32_t (&b0)[3], const uint32_t (&b1)[3])
{
    mma_bf16(c, am, b0[1], b1[1]);
    mma_bf16(c, ah, b0[2], b1[2]);
    mma_bf16(c, al, b0[0], b1[0]);
    mma_bf16(c, ah, b0[1], b1[1]);
    mma_bf16(c, am, b0[0], b1[0]);
    mma_bf16(c, ah, b0[0], b1[0]);
}

// a float4 as three planes of four bf16 each
__device__ __forceinline__ void split_store(float4 v, uint8_t *dst, int plane)
{
    __nv_bfloat16 p[3][4];
    split3(v.x, p[0][0], p[1][0], p[2][0]), split3(v.y, p[0][1], p[1][1], p[2][1]);
    split3(v.z, p[0][2], p[1][2], p[2][2]), split3(v.w, p[0][3], p[1][3], p[2][3]);
#pragma unroll
    for (int pl = 0; pl < 3; ++pl) *reinterpret_cast<uint2 *>(dst + pl * plane) = make_uint2(pack2(p[pl][0], p[pl][1]), pack2(p[pl][2], p[pl][3]));
}

// S = Q K^T of 16 rows x 16 NP keys; qa / ka: this lane's ldmatrix addresses in the first planes
template <int HD, int NP>
__device__ __forceinline__ void scores_of_tile(uint32_t qa, int qplane, uint32_t ka, int kplane, float (&s)[2 * NP][4])
{
    float s2[2 * NP][4];  // s, s2: even and odd k-steps: two independent chains of dependent MMAs per key tile
#pragma unroll
    for (int n = 0; n < 2 * NP; ++n) s[n][0] = s[n][1] = s[n][2] = s[n][3] = s2[n][0] = s2[n][1] = s2[n][2] = s2[n][3] = 0.f;
#pragma unroll
    for (int ks = 0; ks < HD / 16; ++ks) {
        uint32_t ah[4], am[4], al[4];
        ldsm4(qa + 32 * ks, ah);
        ldsm4(qa + qplane + 32 * ks, am);
        ldsm4(qa + 2 * qplane + 32 * ks, al);
#pragma unroll
        for (int np = 0; np < NP; ++np) {  // two key tiles per ldmatrix
            uint32_t b[3][4];
#pragma unroll
            for (int pl = 0; pl < 3; ++pl) ldsm4(ka + pl * kplane + np * 16 * (HD * 2 + 16) + 32 * ks, b[pl]);
            const uint32_t b0a[3] = {b[0][0], b[1][0], b[2][0]}, b1a[3] = {b[0][1], b[1][1], b[2][1]};
            const uint32_t b0b[3] = {b[0][2], b[1][2], b[2][2]}, b1b[3] = {b[0][3], b[1][3], b[2][3]};
            if (ks & 1) {
                mma6(s2[2 * np], ah, am, al, b0a, b1a);
                mma6(s2[2 * np + 1], ah, am, al, b0b, b1b);
            } else {
                mma6(s[2 * np], ah, am, al, b0a, b1a);
                mma6(s[2 * np + 1], ah, am, al, b0b, b1b);
            }
        }
    }
#pragma unroll
    for (int n = 0; n < 2 * NP; ++n) s[n][0] += s2[n][0], s[n][1] += s2[n][1], s[n][2] += s2[n][2], s[n][3] += s2[n][3];
}

// scaled scores, -inf past the keys that rows g (len0) and g + 8 (len1) see, and the rows' maxima; key0: this lane's first key
template <int NN>
__device__ __forceinline__ void mask_scores(float (&s)[NN][4], int key0, int len0, int len1, float scale, float &tm0, float &tm1)
{
    tm0 = -INFINITY, tm1 = -INFINITY;
#pragma unroll
    for (int n = 0; n < NN; ++n) {
        const int key = key0 + 8 * n;
        s[n][0] = key < len0 ? s[n][0] * scale : -INFINITY, s[n][1] = key + 1 < len0 ? s[n][1] * scale : -INFINITY;
        s[n][2] = key < len1 ? s[n][2] * scale : -INFINITY, s[n][3] = key + 1 < len1 ? s[n][3] * scale : -INFINITY;
        tm0 = fmaxf(tm0, fmaxf(s[n][0], s[n][1])), tm1 = fmaxf(tm1, fmaxf(s[n][2], s[n][3]));
    }
    tm0 = fmaxf(tm0, __shfl_xor_sync(0xffffffffu, tm0, 1)), tm0 = fmaxf(tm0, __shfl_xor_sync(0xffffffffu, tm0, 2));
    tm1 = fmaxf(tm1, __shfl_xor_sync(0xffffffffu, tm1, 1)), tm1 = fmaxf(tm1, __shfl_xor_sync(0xffffffffu, tm1, 2));
}

// P = exp(s - new maximum) as split A operands, the correction exp(old - new maximum) and the tile's row sums
__device__ __forceinline__ void weights_of_tile(const float (&s)[KT / 8][4], float m0, float m1, float nm0, float nm1, float &c0, float &c1, float &ps0,
                                                float &ps1, uint32_t (&ph)[KT / 16][4], uint32_t (&pm)[KT / 16][4], uint32_t (&pl)[KT / 16][4])
{
    // a row that sees no key of this tile (and none before) keeps m = -inf: its weights and corrections are 0
    c0 = nm0 > -INFINITY ? expf(m0 - nm0) : 0.f, c1 = nm1 > -INFINITY ? expf(m1 - nm1) : 0.f;
    ps0 = 0.f, ps1 = 0.f;
#pragma unroll
    for (int n = 0; n < KT / 8; ++n) {
        float p[4];
        p[0] = nm0 > -INFINITY ? expf(s[n][0] - nm0) : 0.f, p[1] = nm0 > -INFINITY ? expf(s[n][1] - nm0) : 0.f;
        p[2] = nm1 > -INFINITY ? expf(s[n][2] - nm1) : 0.f, p[3] = nm1 > -INFINITY ? expf(s[n][3] - nm1) : 0.f;
        ps0 += p[0] + p[1], ps1 += p[2] + p[3];
        __nv_bfloat16 hi[4], mi[4], lo[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) split3(p[i], hi[i], mi[i], lo[i]);
        // accumulator (row g: cols 2tg, 2tg+1 | row g+8) of key tile n -> A regs: tile 2j -> a0 (row g), a1 (row g+8); tile 2j+1 -> a2, a3
        const int j = n >> 1, o2 = (n & 1) * 2;
        ph[j][o2] = pack2(hi[0], hi[1]), ph[j][o2 + 1] = pack2(hi[2], hi[3]);
        pm[j][o2] = pack2(mi[0], mi[1]), pm[j][o2 + 1] = pack2(mi[2], mi[3]);
        pl[j][o2] = pack2(lo[0], lo[1]), pl[j][o2 + 1] = pack2(lo[2], lo[3]);
    }
    ps0 += __shfl_xor_sync(0xffffffffu, ps0, 1), ps0 += __shfl_xor_sync(0xffffffffu, ps0, 2);
    ps1 += __shfl_xor_sync(0xffffffffu, ps1, 1), ps1 += __shfl_xor_sync(0xffffffffu, ps1, 2);
}

// Shared memory (bf16 planes, plane p of a tile at p * rows * LDB bytes): Q [3][HPC * 64][LD], K [3][32][LD], V [3][32][LD]
// Q8: the cache holds Q8_0 rows as int8 planes kc / vc [.., maxSeq, HD] with fp16 block scales kd / vd [.., maxSeq, HD / 32]
// (QuantizedKVCache); a staged value is d * q, a 19-bit number that its three bf16 parts hold exactly, so the contraction
// sees exactly what ScaledDotProductFlashQ8_0* reads from the cache (AttentionKernels.cs:489-813).
template <int HD, int HPC, bool Q8>
__global__ void __launch_bounds__(128 * HPC) sdpa_prefill_mma_kernel(const float *__restrict__ q, const void *__restrict__ kc,
                                                                     const void *__restrict__ vc, const __half *__restrict__ kd,
                                                                     const __half *__restrict__ vd, float *__restrict__ out, int T,
                                                                     int nh, int nkv, int pos0, int maxSeq, float scale)
{
    constexpr int LDB = HD * 2 + 16;                 // bytes per row of a plane
    constexpr int QPLANE = HPC * QROWS * LDB, KPLANE = KT * LDB;
    constexpr int NTH = 128 * HPC;
    extern __shared__ __align__(16) uint8_t sm_raw[];
    uint8_t *sq = sm_raw, *sk = sq + 3 * QPLANE, *sv = sk + 3 * KPLANE;
    const uint32_t sq_a = (uint32_t)__cvta_generic_to_shared(sq), sk_a = (uint32_t)__cvta_generic_to_shared(sk),
                   sv_a = (uint32_t)__cvta_generic_to_shared(sv);
    smc_grid_dep_sync();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, tg = lane & 3;
    const int hl = warp >> 2, wq = warp & 3;          // head of the CTA's group, 16-row slice of the 64 rows
    const int hg = blockIdx.x;                          // head group; the grid's fast index, so CTAs start heaviest tile first
    const int h = hg * HPC + hl, kvh = (hg * HPC) / (nh / nkv);
    const int t0 = (int)(gridDim.y - 1 - blockIdx.y) * QROWS;  // later rows see more keys: they start first
    const int cta_len = pos0 + min(T, t0 + QROWS);    // keys any row of this CTA sees
    const float *kbase = static_cast<const float *>(kc) + (size_t)kvh * maxSeq * HD, *vbase = static_cast<const float *>(vc) + (size_t)kvh * maxSeq * HD;
    const int8_t *kqb = static_cast<const int8_t *>(kc) + (size_t)kvh * maxSeq * HD, *vqb = static_cast<const int8_t *>(vc) + (size_t)kvh * maxSeq * HD;
    const __half *kdb = Q8 ? kd + (size_t)kvh * maxSeq * (HD / 32) : nullptr, *vdb = Q8 ? vd + (size_t)kvh * maxSeq * (HD / 32) : nullptr;

    // ---- Q: split once
    for (int e = threadIdx.x; e < HPC * QROWS * (HD / 4); e += NTH) {
        const int c = e % (HD / 4), r = (e / (HD / 4)) % QROWS, hh = e / (QROWS * (HD / 4));
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t0 + r < T) v = *reinterpret_cast<const float4 *>(q + ((size_t)(t0 + r) * nh + hg * HPC + hh) * HD + 4 * c);
        __nv_bfloat16 p[3][4];
        split3(v.x, p[0][0], p[1][0], p[2][0]), split3(v.y, p[0][1], p[1][1], p[2][1]);
        split3(v.z, p[0][2], p[1][2], p[2][2]), split3(v.w, p[0][3], p[1][3], p[2][3]);
#pragma unroll
        for (int pl = 0; pl < 3; ++pl)
            *reinterpret_cast<uint2 *>(sq + pl * QPLANE + (hh * QROWS + r) * LDB + 8 * c) = make_uint2(pack2(p[pl][0], p[pl][1]), pack2(p[pl][2], p[pl][3]));
    }

    // rows of this lane: g and g + 8 of the warp's 16
    const int row0 = t0 + wq * 16 + g, row1 = row0 + 8;
    const int len0 = row0 < T ? pos0 + row0 + 1 : 0, len1 = row1 < T ? pos0 + row1 + 1 : 0;  // keys each row sees
    const int warp_len = t0 + wq * 16 < T ? pos0 + min(T, t0 + wq * 16 + 16) : 0;
    float o[HD / 8][4];
#pragma unroll
    for (int n = 0; n < HD / 8; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;

    // ldmatrix lane addressing
    const uint32_t a_off = (uint32_t)((hl * QROWS + wq * 16 + (lane & 7) + 8 * ((lane >> 3) & 1)) * LDB + 16 * (lane >> 4));
    const uint32_t bk_off = (uint32_t)(((lane & 7) + 8 * (lane >> 4)) * LDB + 16 * ((lane >> 3) & 1));   // K: [key][dim], two key tiles
    const uint32_t bv_off = (uint32_t)(((lane & 7) + 8 * ((lane >> 3) & 1)) * LDB + 16 * (lane >> 4));   // V: transposed, two dim tiles

    // A tile's K and V rows are requested one iteration ahead into registers (the loads fly while the previous tile is
    // multiplied), then split into their planes and stored once everybody has finished reading that previous tile.
    constexpr int PF = KT * (HD / 4) / NTH;  // float4 pieces of K (and of V) per thread and tile
    float4 pk[PF], pv[PF];
    auto fetch = [&](int start) {
#pragma unroll
        for (int i = 0; i < PF; ++i) {
            const int e = threadIdx.x + i * NTH, r = e / (HD / 4), c = e % (HD / 4);
            pk[i] = pv[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (start + r < cta_len) {
                if (Q8) {  // four codes and their block's scale: the piece is d * q
                    const size_t row = (size_t)(start + r);
                    const char4 ck = *reinterpret_cast<const char4 *>(kqb + row * HD + 4 * c), cv = *reinterpret_cast<const char4 *>(vqb + row * HD + 4 * c);
                    const float dk = __half2float(kdb[row * (HD / 32) + c / 8]), dv = __half2float(vdb[row * (HD / 32) + c / 8]);
                    pk[i] = make_float4(dk * (float)ck.x, dk * (float)ck.y, dk * (float)ck.z, dk * (float)ck.w);
                    pv[i] = make_float4(dv * (float)cv.x, dv * (float)cv.y, dv * (float)cv.z, dv * (float)cv.w);
                } else {
                    pk[i] = *reinterpret_cast<const float4 *>(kbase + (size_t)(start + r) * HD + 4 * c);
                    pv[i] = *reinterpret_cast<const float4 *>(vbase + (size_t)(start + r) * HD + 4 * c);
                }
            }
        }
    };
    auto stash = [&]() {
#pragma unroll
        for (int i = 0; i < PF; ++i) {
            const int e = threadIdx.x + i * NTH, r = e / (HD / 4), c = e % (HD / 4);
            __nv_bfloat16 p[3][4];
            split3(pk[i].x, p[0][0], p[1][0], p[2][0]), split3(pk[i].y, p[0][1], p[1][1], p[2][1]);
            split3(pk[i].z, p[0][2], p[1][2], p[2][2]), split3(pk[i].w, p[0][3], p[1][3], p[2][3]);
#pragma unroll
            for (int pl = 0; pl < 3; ++pl)
                *reinterpret_cast<uint2 *>(sk + pl * KPLANE + r * LDB + 8 * c) = make_uint2(pack2(p[pl][0], p[pl][1]), pack2(p[pl][2], p[pl][3]));
            split3(pv[i].x, p[0][0], p[1][0], p[2][0]), split3(pv[i].y, p[0][1], p[1][1], p[2][1]);
            split3(pv[i].z, p[0][2], p[1][2], p[2][2]), split3(pv[i].w, p[0][3], p[1][3], p[2][3]);
#pragma unroll
            for (int pl = 0; pl < 3; ++pl)
                *reinterpret_cast<uint2 *>(sv + pl * KPLANE + r * LDB + 8 * c) = make_uint2(pack2(p[pl][0], p[pl][1]), pack2(p[pl][2], p[pl][3]));
        }
    };
    fetch(0);
    for (int start = 0; start < cta_len; start += KT) {
        __syncthreads();  // the previous tile has been consumed (and Q is in place before its first use)
        stash();
        __syncthreads();
        if (start + KT < cta_len) fetch(start + KT);  // in flight under this tile's MMAs
        if (start >= warp_len) continue;  // warp uniform: every row's causal bound lies before the tile

        // ---- S = Q K^T for 16 rows x 32 keys
        float s[KT / 8][4];
        scores_of_tile<HD, KT / 16>(sq_a + a_off, QPLANE, sk_a + bk_off, KPLANE, s);
        // ---- online softmax: lane holds keys start + 8n + 2tg, + 1 of rows g (s[n][0..1]) and g + 8 (s[n][2..3])
        float tm0, tm1;
        mask_scores<KT / 8>(s, start + 2 * tg, len0, len1, scale, tm0, tm1);
        const float nm0 = fmaxf(m0, tm0), nm1 = fmaxf(m1, tm1);
        float c0, c1, ps0, ps1;
        uint32_t ph[KT / 16][4], pm[KT / 16][4], pl_[KT / 16][4];  // P as A operands: k16 = two key tiles
        weights_of_tile(s, m0, m1, nm0, nm1, c0, c1, ps0, ps1, ph, pm, pl_);
        l0 = fmaf(l0, c0, ps0), l1 = fmaf(l1, c1, ps1);
        m0 = nm0, m1 = nm1;
#pragma unroll
        for (int n = 0; n < HD / 8; ++n) o[n][0] *= c0, o[n][1] *= c0, o[n][2] *= c1, o[n][3] *= c1;
        // ---- O += P V
#pragma unroll
        for (int j = 0; j < KT / 16; ++j) {
#pragma unroll
            for (int np = 0; np < HD / 16; ++np) {  // two dim tiles per ldmatrix
                uint32_t b[3][4];
#pragma unroll
                for (int pl = 0; pl < 3; ++pl) ldsm4t(sv_a + pl * KPLANE + bv_off + j * 16 * LDB + 32 * np, b[pl]);
                const uint32_t b0a[3] = {b[0][0], b[1][0], b[2][0]}, b1a[3] = {b[0][1], b[1][1], b[2][1]};
                const uint32_t b0b[3] = {b[0][2], b[1][2], b[2][2]}, b1b[3] = {b[0][3], b[1][3], b[2][3]};
                mma6(o[2 * np], ph[j], pm[j], pl_[j], b0a, b1a);
                mma6(o[2 * np + 1], ph[j], pm[j], pl_[j], b0b, b1b);
            }
        }
    }
    // ---- out = O / l
    const float i0 = l0 > 0.f ? 1.0f / l0 : 0.f, i1 = l1 > 0.f ? 1.0f / l1 : 0.f;
#pragma unroll
    for (int n = 0; n < HD / 8; ++n) {
        if (row0 < T) *reinterpret_cast<float2 *>(out + ((size_t)row0 * nh + h) * HD + 8 * n + 2 * tg) = make_float2(o[n][0] * i0, o[n][1] * i0);
        if (row1 < T) *reinterpret_cast<float2 *>(out + ((size_t)row1 * nh + h) * HD + 8 * n + 2 * tg) = make_float2(o[n][2] * i1, o[n][3] * i1);
    }
}

// ------------------------------------------------------------------------------ few rows over a long cache
// Up to 16 query rows (a draft's tokens) over an fp32 cache: the kernel above gives every head pair one CTA, whose two busy
// warps walk the cache's tiles one after the other (5 us a tile: 384 dependent MMAs, exponentials, staging).  Here a cluster of
// HD / 16 CTAs shares one head pair and eight rows, and cuts that walk by what its steps depend on, so that every sum is still
// formed by the same MMAs in the same order and every output keeps its bits:
//   1. scores and tile maxima: tiles are independent; CTA r takes tiles r, r + CS, ..., a warp per head and half tile
//   2. with all tile maxima known (they go to every CTA of the cluster) the running maximum before and after a tile is a
//      maximum over earlier tiles: weights, corrections and row sums of all tiles at once
//   3. only O += P V and l follow the tiles in order; CTA r does it for one head and 32 output dims, a warp for 8 of them, while the other four warps
//      bring V and the weights, those from the CTA that made them through distributed shared memory
// Shared memory stays below half an SM's: with one CTA per SM fewer than 16 clusters of eight were resident at once, and the
// 16 head pairs of a 32-head model took two waves.  What bounds it: step 1's MMAs, and step 3's rounds of three tiles.  When a CTA did 16 dims of
// both heads and its MMA warps read the weights themselves, all CTAs of the cluster read the weights of a tile of both heads from the same CTA at the
// same time, and 280 bytes of a thread's registers were spilled.
// Six rows over 1021 keys, 32 heads on 8 KV heads of 128, one layer: 175 us in the kernel above, 43 -> 33 us here (101 keys 16 -> 13, 2200 keys 78 -> 55);
// a 32-layer pass of six rows 3557 -> 3241 us, of a small model's 28 layers 1601 -> 1334.  (The request into L2 ahead of the predecessor's end is 0.5 and 5 % of that.)
// Scores and weights of all of a CTA's tiles are kept in shared memory, which ends at 14 tiles: 3584 keys at head size 128, 1792 at 64.
// Longer caches go to the tcgen05 prompt kernel, as do Q8_0 caches and groups of an odd number of heads.
constexpr int FEW_ROWS = 8;  // per cluster: rows 8 .. 15 of the MMAs are not used
template <int HD>
struct FewShape {
    static constexpr int CS = HD / 16, LDB = HD * 2 + 16;
    static constexpr int LOCAL = 14, TILES = LOCAL * CS;  // key tiles of one CTA, and in all
    static constexpr int QPLANE = 2 * FEW_ROWS * LDB, KPLANE = 2 * KT * LDB, S_JOB = 1024, P_JOB = 3 * 512;
    static constexpr int V_LD = 80, V_TILES = 3, V_KEYS = V_TILES * KT, VPLANE = V_KEYS * V_LD;  // 32 dims of a key: 64 bytes, padded to an odd multiple of 16
    // Q and K, then scores; later weights where Q and K were, then two stages of V and of the weights it meets over the rest and the scores
    static constexpr int QK = 3 * (QPLANE + KPLANE) > 2 * LOCAL * P_JOB ? 3 * (QPLANE + KPLANE) : 2 * LOCAL * P_JOB;
    static constexpr int OFF_K = 3 * QPLANE, OFF_S = QK, OFF_P = 0, OFF_V = 2 * LOCAL * P_JOB, OFF_W = OFF_V + 2 * 3 * VPLANE, W_END = OFF_W + 2 * V_TILES * P_JOB;
    static constexpr int END = OFF_S + 2 * LOCAL * S_JOB > W_END ? OFF_S + 2 * LOCAL * S_JOB : W_END;
    static constexpr int OFF_TM = END, OFF_CP = OFF_TM + 2 * 2 * TILES * FEW_ROWS * 4, OFF_WC = OFF_CP + 2 * LOCAL * FEW_ROWS * 8;
    static constexpr int SMEM = OFF_WC + 2 * V_TILES * FEW_ROWS * 8;
    static_assert(SMEM <= 113 * 1024, "two CTAs per SM");
};
__device__ __forceinline__ void prefetch_l2(const void *src, uint32_t bytes)
{
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ uint32_t cluster_map(uint32_t addr, uint32_t cta)
{
    uint32_t v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(v) : "r"(addr), "r"(cta));
    return v;
}
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int HD>
__global__ void __launch_bounds__(256, 2) sdpa_few_rows_kernel(const float *__restrict__ q, const float *__restrict__ kc, const float *__restrict__ vc,
                                                               float *__restrict__ out, int T, int nh, int nkv, int pos0, int maxSeq, float scale)
{
    using S = FewShape<HD>;
    constexpr int LDB = S::LDB, CS = S::CS;
    extern __shared__ __align__(16) uint8_t sm_raw[];
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(sm_raw);
    float2 *sc = reinterpret_cast<float2 *>(sm_raw + S::OFF_S);              // scores of row g [job][4][lane]
    uint4 *sp = reinterpret_cast<uint4 *>(sm_raw + S::OFF_P);                // weights of row g [job][plane][lane]
    const float *tmx = reinterpret_cast<const float *>(sm_raw + S::OFF_TM);  // maxima [head][half tile][row]
    float2 *cp = reinterpret_cast<float2 *>(sm_raw + S::OFF_CP);             // (correction, row sum) [job][row]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, tg = lane & 3;
    const int hg = blockIdx.x / CS, rank = blockIdx.x % CS, kvh = hg * 2 / (nh / nkv), t0 = (int)blockIdx.y * FEW_ROWS;
    const int len = pos0 + T, tiles = (len + KT - 1) / KT, local = tiles > rank ? (tiles - rank + CS - 1) / CS : 0;
    const float *kbase = kc + (size_t)kvh * maxSeq * HD, *vbase = vc + (size_t)kvh * maxSeq * HD;
    // The keys and values that are there already are asked for, into L2, before the predecessor is waited for (it writes the newest rows, to L2).
    if (threadIdx.x == 0) {
        const int part = (pos0 + CS - 1) / CS, k0 = rank * part, n = min(pos0, k0 + part) - k0;
        if (n > 0) prefetch_l2(kbase + (size_t)k0 * HD, (uint32_t)n * HD * 4), prefetch_l2(vbase + (size_t)k0 * HD, (uint32_t)n * HD * 4);
    }
    smc_grid_dep_sync();

    constexpr int PF = 2 * KT * (HD / 4) / 256;  // K: two tiles at a time, requested before the previous two are multiplied
    float4 pk[PF];
    auto fetch_k = [&](int lt0) {
#pragma unroll
        for (int i = 0; i < PF; ++i) {
            const int e = threadIdx.x + i * 256, r = e / (HD / 4), c = e % (HD / 4);
            const int key = ((lt0 + r / KT) * CS + rank) * KT + r % KT;
            pk[i] = key < len ? *reinterpret_cast<const float4 *>(kbase + (size_t)key * HD + 4 * c) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    fetch_k(0);
    for (int e = threadIdx.x; e < 2 * FEW_ROWS * (HD / 4); e += 256) {  // Q: split once
        const int c = e % (HD / 4), r = (e / (HD / 4)) % FEW_ROWS, hh = e / (FEW_ROWS * (HD / 4));
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t0 + r < T) v = *reinterpret_cast<const float4 *>(q + ((size_t)(t0 + r) * nh + hg * 2 + hh) * HD + 4 * c);
        split_store(v, sm_raw + (hh * FEW_ROWS + r) * LDB + 8 * c, S::QPLANE);
    }
    cluster_sync();  // every CTA of the cluster runs: its shared memory may be written
    const int len0 = t0 + g < T ? pos0 + t0 + g + 1 : 0;  // keys that row g sees

    // ---- 1: scores of this CTA's tiles, two at a time
    {
        const int hl = warp >> 2, tl = (warp >> 1) & 1, np = warp & 1;
        // rows 8 .. 15 of the A operand come from the same addresses as rows 0 .. 7: what they yield is not used
        const uint32_t qa = base + (uint32_t)((hl * FEW_ROWS + (lane & 7)) * LDB + 16 * (lane >> 4));
        const uint32_t ka = base + S::OFF_K + (uint32_t)((tl * KT + np * 16 + (lane & 7) + 8 * (lane >> 4)) * LDB + 16 * ((lane >> 3) & 1));
        for (int lt0 = 0; lt0 < local; lt0 += 2) {
            __syncthreads();  // the previous two tiles have been read
#pragma unroll
            for (int i = 0; i < PF; ++i) {
                const int e = threadIdx.x + i * 256, r = e / (HD / 4), c = e % (HD / 4);
                split_store(pk[i], sm_raw + S::OFF_K + r * LDB + 8 * c, S::KPLANE);
            }
            __syncthreads();
            if (lt0 + 2 < local) fetch_k(lt0 + 2);
            const int lt = lt0 + tl, tile = lt * CS + rank;
            if (lt >= local) continue;  // warp uniform
            float s[2][4];
            scores_of_tile<HD, 1>(qa, S::QPLANE, ka, S::KPLANE, s);
            float tm0, tm1;
            mask_scores<2>(s, tile * KT + np * 16 + 2 * tg, len0, 0, scale, tm0, tm1);
            const int job = hl * S::LOCAL + lt;
#pragma unroll
            for (int n = 0; n < 2; ++n) sc[(job * 4 + 2 * np + n) * 32 + lane] = make_float2(s[n][0], s[n][1]);
            const uint32_t at = base + S::OFF_TM + 4u * (uint32_t)((hl * 2 * S::TILES + 2 * tile + np) * FEW_ROWS + g);
            for (int cta = tg; cta < CS; cta += 4)
                asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(cluster_map(at, (uint32_t)cta)), "f"(tm0) : "memory");
        }
    }
    cluster_sync();
    // ---- 2: weights, corrections and row sums of this CTA's tiles
    for (int j = warp; j < 2 * local; j += 8) {
        const int hl = j & 1, lt = j >> 1, tile = lt * CS + rank, job = hl * S::LOCAL + lt;
        const float *tmh = tmx + hl * 2 * S::TILES * FEW_ROWS + g;
        float m0 = -INFINITY;
        for (int t = tg; t < 2 * tile; t += 4) m0 = fmaxf(m0, tmh[t * FEW_ROWS]);
        m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, 1)), m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, 2));
        const float nm0 = fmaxf(m0, fmaxf(tmh[2 * tile * FEW_ROWS], tmh[(2 * tile + 1) * FEW_ROWS]));
        float s[KT / 8][4];
#pragma unroll
        for (int n = 0; n < KT / 8; ++n) {
            const float2 v = sc[(job * 4 + n) * 32 + lane];
            s[n][0] = v.x, s[n][1] = v.y, s[n][2] = s[n][3] = -INFINITY;
        }
        float c0, c1, ps0, ps1;
        uint32_t ph[KT / 16][4], pm[KT / 16][4], pl[KT / 16][4];
        weights_of_tile(s, m0, -INFINITY, nm0, -INFINITY, c0, c1, ps0, ps1, ph, pm, pl);
        uint4 *dst = sp + job * 3 * 32 + lane;
        dst[0] = make_uint4(ph[0][0], ph[0][2], ph[1][0], ph[1][2]);
        dst[32] = make_uint4(pm[0][0], pm[0][2], pm[1][0], pm[1][2]);
        dst[64] = make_uint4(pl[0][0], pl[0][2], pl[1][0], pl[1][2]);
        if (tg == 0) cp[job * FEW_ROWS + g] = make_float2(c0, ps0);
    }
    // ---- 3: O and l in tile order, one head and 32 dims per CTA: four warps of 8 dims multiply, the other four bring V and the weights, a chunk of
    // V_TILES tiles ahead in shared memory and another in registers
    const int hl3 = rank / (CS / 2), d3 = rank % (CS / 2) * 32;
    constexpr int PIECES = S::V_KEYS * 8, WORDS = S::V_TILES * (S::P_JOB / 16), ROWS3 = S::V_TILES * FEW_ROWS;
    auto load_v = [&](int e, int chunk) {  // four dims of a key
        const int key = chunk * S::V_KEYS + e / 8;
        return e < PIECES && key < len ? *reinterpret_cast<const float4 *>(vbase + (size_t)key * HD + d3 + 4 * (e & 7)) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    auto store_v = [&](int e, int chunk, const float4 &v) {
        if (e < PIECES) split_store(v, sm_raw + S::OFF_V + (chunk & 1) * 3 * S::VPLANE + (e / 8) * S::V_LD + 8 * (e & 7), S::VPLANE);
    };
    auto load_w = [&](int e, int chunk, uint4 &v) {  // 16 bytes of a tile's weights, from the CTA that made them
        const int tile = chunk * S::V_TILES + e / (S::P_JOB / 16);
        if (e >= WORDS || tile >= tiles) return;
        const uint32_t at = cluster_map(base + S::OFF_P, (uint32_t)(tile % CS)) + (uint32_t)((hl3 * S::LOCAL + tile / CS) * S::P_JOB + 16 * (e % (S::P_JOB / 16)));
        asm volatile("ld.shared::cluster.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at) : "memory");
    };
    auto store_w = [&](int e, int chunk, const uint4 &v) {
        if (e < WORDS) *reinterpret_cast<uint4 *>(sm_raw + S::OFF_W + (chunk & 1) * S::V_TILES * S::P_JOB + 16 * e) = v;
    };
    auto load_c = [&](int e, int chunk, float2 &v) {  // (correction, row sum) of a tile's row
        const int tile = chunk * S::V_TILES + e / FEW_ROWS;
        if (e >= ROWS3 || tile >= tiles) return;
        const uint32_t at = cluster_map(base + S::OFF_CP, (uint32_t)(tile % CS)) + 8u * (uint32_t)((hl3 * S::LOCAL + tile / CS) * FEW_ROWS + e % FEW_ROWS);
        asm volatile("ld.shared::cluster.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(at) : "memory");
    };
    auto store_c = [&](int e, int chunk, const float2 &v) {
        if (e < ROWS3) *reinterpret_cast<float2 *>(sm_raw + S::OFF_WC + 8 * ((chunk & 1) * ROWS3 + e)) = v;
    };
    auto bring = [&](auto threads, int t, auto request, auto keep) {
        constexpr int TH = decltype(threads)::value, NV = (PIECES + TH - 1) / TH, NW = (WORDS + TH - 1) / TH;
        float4 v[NV];
        uint4 w[NW];
        float2 c = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < NW; ++i) w[i] = make_uint4(0u, 0u, 0u, 0u);
        auto load = [&](int chunk) {
#pragma unroll
            for (int i = 0; i < NV; ++i) v[i] = load_v(t + i * TH, chunk);
            request();
#pragma unroll
            for (int i = 0; i < NW; ++i) load_w(t + i * TH, chunk, w[i]);
            load_c(t, chunk, c);
        };
        auto store = [&](int chunk) {
#pragma unroll
            for (int i = 0; i < NV; ++i) store_v(t + i * TH, chunk, v[i]);
#pragma unroll
            for (int i = 0; i < NW; ++i) store_w(t + i * TH, chunk, w[i]);
            store_c(t, chunk, c);
        };
        keep(load, store);
    };
    const int chunks = (tiles + S::V_TILES - 1) / S::V_TILES;
    // all warps: chunk 0.  Between its two requests the weights are waited for; nobody needs its scores any more then, and V goes there.
    bring(std::integral_constant<int, 256>{}, threadIdx.x, [] { cluster_sync(); }, [&](auto &load, auto &store) { load(0), store(0); });
    if (warp >= 4) {
        bring(std::integral_constant<int, 128>{}, threadIdx.x - 128, [] {}, [&](auto &load, auto &store) {
            load(1);
            for (int chunk = 0; chunk < chunks; ++chunk) {
                __syncthreads();  // this chunk is staged and the other buffers have been read
                if (chunk + 1 < chunks) store(chunk + 1), load(chunk + 2);
            }
        });
    } else {
        float o[4] = {0.f, 0.f, 0.f, 0.f}, l0 = 0.f;
        struct Operands {
            uint32_t v[3][4];  // [plane][8 keys]
            uint4 w[3];
            float2 c;
        } x[2];  // a tile's; the next one's are fetched before this one's MMAs
        const uint32_t va = base + S::OFF_V + (uint32_t)(lane * S::V_LD + 16 * warp);
        int next = 0, next_chunk = 0;  // the tile to be fetched: its place in its chunk, and the chunk
        auto fetch = [&](Operands &d) {
            if (next == 0) __syncthreads();  // the chunk is staged, and all of the one before it is in registers
            const int buf = next_chunk & 1;
#pragma unroll
            for (int pl = 0; pl < 3; ++pl) {
                ldsm4t(va + (uint32_t)((buf * 3 + pl) * S::VPLANE + next * KT * S::V_LD), d.v[pl]);
                d.w[pl] = *reinterpret_cast<const uint4 *>(sm_raw + S::OFF_W + (buf * S::V_TILES + next) * S::P_JOB + 512 * pl + 16 * lane);
            }
            d.c = *reinterpret_cast<const float2 *>(sm_raw + S::OFF_WC + 8 * (buf * ROWS3 + next * FEW_ROWS + g));
            if (++next == S::V_TILES) next = 0, ++next_chunk;
        };
        auto add = [&](const Operands &d) {
            l0 = fmaf(l0, d.c.x, d.c.y);
            o[0] *= d.c.x, o[1] *= d.c.x;
#pragma unroll
            for (int j = 0; j < KT / 16; ++j) {
                const uint32_t ph[4] = {j ? d.w[0].z : d.w[0].x, 0u, j ? d.w[0].w : d.w[0].y, 0u}, pm[4] = {j ? d.w[1].z : d.w[1].x, 0u, j ? d.w[1].w : d.w[1].y, 0u},
                               pl[4] = {j ? d.w[2].z : d.w[2].x, 0u, j ? d.w[2].w : d.w[2].y, 0u};
                const uint32_t b0[3] = {d.v[0][2 * j], d.v[1][2 * j], d.v[2][2 * j]}, b1[3] = {d.v[0][2 * j + 1], d.v[1][2 * j + 1], d.v[2][2 * j + 1]};
                mma6(o, ph, pm, pl, b0, b1);
            }
        };
        fetch(x[0]);
        for (int tile = 0; tile < tiles; tile += 2) {
            if (tile + 1 < tiles) fetch(x[1]);
            add(x[0]);
            if (tile + 1 >= tiles) break;
            if (tile + 2 < tiles) fetch(x[0]);
            add(x[1]);
        }
        const float i0 = l0 > 0.f ? 1.0f / l0 : 0.f;
        if (t0 + g < T)
            *reinterpret_cast<float2 *>(out + ((size_t)(t0 + g) * nh + hg * 2 + hl3) * HD + d3 + 8 * warp + 2 * tg) = make_float2(o[0] * i0, o[1] * i0);
    }
    cluster_sync();  // nobody leaves while its weights are read
}

}  // namespace

bool smc_sdpa_prefill_mma_supported(int nh, int nkv, int hd) { return (hd == 64 || hd == 128) && nkv > 0 && nh % nkv == 0; }

// kd == null: kc / vc are fp32 rows; else the int8 planes and fp16 block scales of a Q8_0 cache
static int launch_prefill_mma(smc_ctx *ctx, smc_attn_planes *planes, const float *q, const void *kc, const void *vc, const __half *kd, const __half *vd,
                              float *out, int T, int nh, int nkv, int hd, int pos0, int maxSeq, float scale, cudaStream_t s)
{
    const int G = nh / nkv;
    // the order matters: a few rows over a long fp32 cache, then the tcgen05 kernel; all of them give the same bits
    auto go = [&](auto kernel, int hpc) {
        const dim3 grid(nh / hpc, (T + QROWS - 1) / QROWS);
        const size_t ldb = (size_t)hd * 2 + 16;
        const size_t smem = 3 * ((size_t)hpc * QROWS + 2 * KT) * ldb;
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        smc_launch_dep(ctx->use_pdl, kernel, grid, dim3(128 * hpc), smem, s, q, kc, vc, kd, vd, out, T, nh, nkv, pos0, maxSeq, scale);
    };
    const bool two = G % 2 == 0 && ctx->attn_hpc != 1;
    // a few rows over more than a few tiles of an fp32 cache: the same bits from a cluster per head pair and eight rows
    const int tiles = (pos0 + T + KT - 1) / KT;
    if (two && !kd && T <= 2 * FEW_ROWS && tiles >= 4 && tiles <= (hd == 128 ? FewShape<128>::TILES : FewShape<64>::TILES)) {
        auto few = [&](auto kernel, int cs, size_t smem) {
            cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            smc_launch_dep_cluster(ctx->use_pdl, cs, kernel, dim3(nh / 2 * cs, (T + FEW_ROWS - 1) / FEW_ROWS), dim3(256), smem, s, q,
                                   static_cast<const float *>(kc), static_cast<const float *>(vc), out, T, nh, nkv, pos0, maxSeq, scale);
        };
        if (hd == 128) few(sdpa_few_rows_kernel<128>, FewShape<128>::CS, FewShape<128>::SMEM);
        else few(sdpa_few_rows_kernel<64>, FewShape<64>::CS, FewShape<64>::SMEM);
        SMC_LAUNCH_CHECK(ctx);
        return SMC_OK;
    }
    // From so many tiles of keys on tcgen05, two launches.  What the kernels below take grows with the tiles, 2.3 us each at heads of 64 in a CTA of their own to 6 at
    // Q8_0 heads of 128 in pairs, whatever the rows; the other takes 2.4 (heads of 64) or 3.0 us a chunk of two and 7 more.  Measured, us, here / there: heads of
    // 128 in pairs, fp32: 20 keys 10.8 / 13.1, 40 14.1 / 12.4; alone: 40 11.4 / 12.4, 96 with 60 rows 18.3 / 17.8, 128 19.0 / 15.4, Q8_0 40 14.4 / 14.6; heads of 64 in
    // pairs: 64 9.0 / 9.9, 96 11.9 / 12.3, 128 15.0 / 12.2, Q8_0 96 13.4 / 14.5, 128 16.9 / 14.5; alone: 64 7.7 / 9.9, 128 12.4 / 12.3, 160 14.8 / 16.0,
    // 192 17.1 / 14.8, Q8_0 96 12.8 / 14.4, 128 16.1 / 14.3.  Longer: 100 rows behind 1900 keys of a Q8_0 cache, heads of 128 398 / 149; 2048 rows 362 / 164.
    const int first = hd == 128 ? (two || kd ? 2 : 3) : (two || kd ? 4 : 6);
    if (tiles >= first && ctx->attn_hpc != 1 && (reinterpret_cast<uintptr_t>(out) & 15) == 0) {
        const int rc = smc_launch_sdpa_prefill_tc(ctx, planes, q, kc, vc, kd, vd, out, T, nh, nkv, hd, pos0, maxSeq, scale, s);
        if (rc != SMC_E_UNSUPPORTED) return rc;  // else the planes do not reach that far (a very long cache, a full device)
    }
    if (kd) {
        if (hd == 128) two ? go(sdpa_prefill_mma_kernel<128, 2, true>, 2) : go(sdpa_prefill_mma_kernel<128, 1, true>, 1);
        else two ? go(sdpa_prefill_mma_kernel<64, 2, true>, 2) : go(sdpa_prefill_mma_kernel<64, 1, true>, 1);
    } else {
        if (hd == 128) two ? go(sdpa_prefill_mma_kernel<128, 2, false>, 2) : go(sdpa_prefill_mma_kernel<128, 1, false>, 1);
        else two ? go(sdpa_prefill_mma_kernel<64, 2, false>, 2) : go(sdpa_prefill_mma_kernel<64, 1, false>, 1);
    }
    SMC_LAUNCH_CHECK(ctx);
    return SMC_OK;
}

int smc_launch_sdpa_prefill_mma(smc_ctx *ctx, smc_attn_planes *planes, const float *q, const float *kc, const float *vc, float *out, int T, int nh, int nkv,
                                int hd, int pos0, int maxSeq, float scale, cudaStream_t s)
{
    return launch_prefill_mma(ctx, planes, q, kc, vc, nullptr, nullptr, out, T, nh, nkv, hd, pos0, maxSeq, scale, s);
}

// one sequence's Q8_0 cache planes (rows pos0 .. pos0 + T - 1 are the queries' own positions)
int smc_launch_sdpa_prefill_mma_q8(smc_ctx *ctx, smc_attn_planes *planes, const float *q, const int8_t *kq, const __half *kd, const int8_t *vq,
                                   const __half *vd, float *out, int T, int nh, int nkv, int hd, int pos0, int maxSeq, float scale, cudaStream_t s)
{
    return launch_prefill_mma(ctx, planes, q, kq, vq, kd, vd, out, T, nh, nkv, hd, pos0, maxSeq, scale, s);
}
