// Small-batch (2..32 rows, larger batches in passes of 32) quantised-activation matmul on the int8 tensor-core
// path: out[t, r] = sum_blocks (dw * dx) * isum(block) (- the Q4_K min term), the arithmetic of SMC_ACT_Q8.
//
// Why MMA here: with a handful of activation rows the dp4a kernels issue one integer dot per (row, token,
// 4 bytes) and become instruction-bound long before HBM is busy.  One mma.m16n8k32 (s8 x s8 -> s32) covers
// 16 weight rows x 8 tokens x one 32-element block, so the per-block integer sums of 32 rows x 32 tokens cost
// 8 instructions per warp; the per-block scaling (int -> float, dw * dx, fused multiply-add) stays on the
// CUDA cores and is what remains.  Integer block sums are exact, so they equal the dp4a kernels' sums; each
// output adds its scaled block sums in k order within a warp's k range and the eight warps of a CTA (which
// split K) are added in warp order: the result of a row does not depend on the batch size or on the other
// rows (for any batch >= 2; the one-row kernels use a different summation tree).
//
// Three kinds of kernel share these sums, bit for bit:
//   split   Q6_K below 64 rows, and Q8_0 / Q4_K where no other has a better form: a CTA owns 32 weight rows (two m16 tiles) and a pass of tokens, its 8 (16) warps take
//           interleaved k groups and meet in shared memory.  Fragments come straight from global memory as 8-byte words: the dot product does not care
//           about the order of k inside a block, so MMA k index 4*tg + i is bound to byte 8*tg + i and 16 + 4*tg + i to byte 8*tg + 4 + i of the
//           block, for weights and activations alike; a quad of lanes then reads one whole 32-byte sector per row.  Scales are loaded once per
//           lane (lane = row for the weights, lane = token for the activations) and handed round with shuffles.
//   tile    prompt-sized batches of Q8_0 and Q6_K: no split, operands staged in shared memory.
//   staged  2 to 63 rows of Q8_0, small batches of Q4_K: the split, operands staged in shared memory.
#include "smc_common.cuh"

#include <type_traits>

namespace {

constexpr int MMA_ROWS = 32;   // weight rows per CTA
constexpr int MMA_WARPS = 8;
// floats per token of the warps' partial tiles in shared memory: a lane (g, tg) of an accumulator fragment writes token
// 2 * tg (+ 1), row g (+ 8), so 2 * RED_LD = 8 (mod 32) puts the 32 lanes of a store on 32 banks (33 left them 4 deep)
constexpr int RED_LD = 36;

__device__ __forceinline__ void mma_s8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1)
{
    asm(
        "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}

__device__ __forceinline__ uint2 ldg8(const void *p)
{
    uint2 v;
    asm("ld.global.nc.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));  // not volatile: free to be hoisted
    return v;
}

// Adds the warps' partial tiles in warp order and stores out[t, r]; red is [NW warps][TOK tokens][RED_LD], TOK >= 8 * NT.
template <int NT, int NW = MMA_WARPS, int TOK = 32>
__device__ __forceinline__ void reduce_and_store(float (*red)[TOK][RED_LD], const float (&acc)[2][NT][4], float *out, int N, int M,
                                                 int r0, int t0)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, tg = lane & 3;
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int i = 0; i < 4; ++i) red[warp][8 * t + 2 * tg + (i & 1)][mt * 16 + g + ((i >> 1) << 3)] = acc[mt][t][i];
    __syncthreads();
    for (int o = threadIdx.x; o < 32 * 8 * NT; o += blockDim.x) {
        const int row = o & 31, tok = o >> 5;
        float s = red[0][tok][row];
#pragma unroll
        for (int w = 1; w < NW; ++w) s += red[w][tok][row];
        if (r0 + row < N && t0 + tok < M) out[(size_t)(t0 + tok) * N + r0 + row] = s;
    }
    __syncthreads();
}

// ------------------------------------------------------------------------------------------ Q8_0
// Planes: quants [N][K] int8, scales [N][K/32] fp16.  K % 128 == 0; a warp works on groups of four blocks.
// Batches of 64 rows and more that the tile kernel (below) does not take, in passes of 64 tokens that share every weight fragment and scale.
constexpr int Q8_PASS = 64;
__global__ void __launch_bounds__(256, 1)
gemv_mma_q8_0_kernel(const int8_t *__restrict__ wq, const __half *__restrict__ wd, const int8_t *__restrict__ xq,
                     const float *__restrict__ xd, float *__restrict__ out, int N, int K, int M)
{
    constexpr int TOK = Q8_PASS, NT = TOK / 8, XR = TOK / 32;
    extern __shared__ __align__(16) float red_q8[];
    float (*red)[TOK][RED_LD] = reinterpret_cast<float (*)[TOK][RED_LD]>(red_q8);
    smc_grid_dep_sync();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, tg = lane & 3;
    const int r0 = blockIdx.x * MMA_ROWS;
    const int nb = K / 32, ngroups = nb / 4;
    // rows past the end are clamped for loads and masked at the store
    const int8_t *arow[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) arow[j] = wq + (size_t)min(r0 + (j >> 1) * 16 + g + (j & 1) * 8, N - 1) * K + 8 * tg;
    const __half *drow = wd + (size_t)min(r0 + lane, N - 1) * nb;
    {  // one pass of 8 * NT tokens per CTA: blockIdx.y picks the pass (a batch of more than 32 rows fills the grid with passes)
        const int t0 = blockIdx.y * 8 * NT;
        const int8_t *brow[NT];
#pragma unroll
        for (int t = 0; t < NT; ++t) brow[t] = xq + (size_t)min(t0 + 8 * t + g, M - 1) * K + 8 * tg;
        const float *xrow[XR];  // this lane's tokens: lane, and lane + 32 in a 64-token pass
#pragma unroll
        for (int x = 0; x < XR; ++x) xrow[x] = xd + (size_t)min(t0 + 32 * x + lane, M - 1) * nb;
        float acc[2][NT][4];
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int t = 0; t < NT; ++t)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[mt][t][i] = 0.f;
        for (int gi = warp; gi < ngroups; gi += MMA_WARPS) {
            // all weight bytes of the group are requested before any of them is used: 4 KB in flight per warp
            uint2 aq[4][4];
#pragma unroll
            for (int kb = 0; kb < 4; ++kb)
#pragma unroll
                for (int j = 0; j < 4; ++j) aq[kb][j] = ldg8(arow[j] + (gi * 4 + kb) * 32);
            const uint2 dwp = *reinterpret_cast<const uint2 *>(drow + gi * 4);   // this lane's row, 4 blocks
            float4 dxp[XR];                                                      // this lane's tokens, 4 blocks
#pragma unroll
            for (int x = 0; x < XR; ++x) dxp[x] = *reinterpret_cast<const float4 *>(xrow[x] + gi * 4);
#pragma unroll
            for (int kb = 0; kb < 4; ++kb) {
                const int koff = (gi * 4 + kb) * 32;
                uint2 b[NT];
                const uint2 (&a)[4] = aq[kb];
#pragma unroll
                for (int t = 0; t < NT; ++t) b[t] = ldg8(brow[t] + koff);
                const uint32_t dword = (kb & 2) ? dwp.y : dwp.x;
                float dxl[XR];
#pragma unroll
                for (int x = 0; x < XR; ++x) dxl[x] = kb == 0 ? dxp[x].x : kb == 1 ? dxp[x].y : kb == 2 ? dxp[x].z : dxp[x].w;
                float dw[2][2];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint32_t wv = __shfl_sync(0xffffffffu, dword, (j >> 1) * 16 + g + (j & 1) * 8);
                    dw[j >> 1][j & 1] = smc_h2f((uint16_t)((kb & 1) ? (wv >> 16) : (wv & 0xFFFFu)));
                }
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    const float dx0 = __shfl_sync(0xffffffffu, dxl[t >> 2], 8 * (t & 3) + 2 * tg);
                    const float dx1 = __shfl_sync(0xffffffffu, dxl[t >> 2], 8 * (t & 3) + 2 * tg + 1);
#pragma unroll
                    for (int mt = 0; mt < 2; ++mt) {
                        int c[4];
                        mma_s8(c, a[2 * mt].x, a[2 * mt + 1].x, a[2 * mt].y, a[2 * mt + 1].y, b[t].x, b[t].y);
                        acc[mt][t][0] = fmaf((float)c[0], dw[mt][0] * dx0, acc[mt][t][0]);
                        acc[mt][t][1] = fmaf((float)c[1], dw[mt][0] * dx1, acc[mt][t][1]);
                        acc[mt][t][2] = fmaf((float)c[2], dw[mt][1] * dx0, acc[mt][t][2]);
                        acc[mt][t][3] = fmaf((float)c[3], dw[mt][1] * dx1, acc[mt][t][3]);
                    }
                }
            }
        }
        reduce_and_store<NT, MMA_WARPS, TOK>(red, acc, out, N, M, r0, t0);
    }
}

// ------------------------------------------------------------------------------------------ Q4_K
// GGUF blocks of 144 bytes: d, dmin (fp16), 12 packed scale / min bytes, 128 nibble bytes; the 32 bytes of
// group gq hold sub-block 2*gq in the low nibbles and 2*gq + 1 in the high ones.  K % 256 == 0; a warp works
// on whole 256-element blocks.  out += d*sc_j * dx * isum  -  dmin*m_j * (dx * sum(xq))  per sub-block.
// Batches of 17 rows and more, in passes of 32, where the staged kernel (below) has no better form.
__global__ void __launch_bounds__(256, 1)
gemv_mma_q4_K_kernel(const uint8_t *__restrict__ raw, const int8_t *__restrict__ xq, const float *__restrict__ xd,
                     const float *__restrict__ xsd, float *__restrict__ out, int N, int K, int M)
{
    constexpr int NT = 4;
    __shared__ float red[MMA_WARPS][32][RED_LD];
    smc_grid_dep_sync();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, tg = lane & 3;
    const int r0 = blockIdx.x * MMA_ROWS;
    const int nb = K / 32, nsb = K / 256;
    const size_t row_bytes = (size_t)nsb * 144;
    const uint8_t *arow[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) arow[j] = raw + (size_t)min(r0 + (j >> 1) * 16 + g + (j & 1) * 8, N - 1) * row_bytes + 16 + 8 * tg;
    const uint8_t *hrow = raw + (size_t)min(r0 + lane, N - 1) * row_bytes;
    {  // one pass of 8 * NT tokens per CTA: blockIdx.y picks the pass (a batch of more than 32 rows fills the grid with passes)
        const int t0 = blockIdx.y * 8 * NT;
        const int8_t *brow[NT];
#pragma unroll
        for (int t = 0; t < NT; ++t) brow[t] = xq + (size_t)min(t0 + 8 * t + g, M - 1) * K + 8 * tg;
        const float *xrow = xd + (size_t)min(t0 + lane, M - 1) * nb;
        const float *srow = xsd + (size_t)min(t0 + lane, M - 1) * nb;
        float acc[2][NT][4];
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int t = 0; t < NT; ++t)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[mt][t][i] = 0.f;
        for (int sb = warp; sb < nsb; sb += MMA_WARPS) {
            // this lane's row: d * sc_j and dmin * m_j of the eight sub-blocks
            const uint4 hdr = *reinterpret_cast<const uint4 *>(hrow + (size_t)sb * 144);
            const float d = smc_h2f((uint16_t)(hdr.x & 0xFFFFu)), dmin = smc_h2f((uint16_t)(hdr.x >> 16));
            float dsc[8], dmn[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                int sc, mn;
                smc_k4_scale_min(hdr.y, hdr.z, hdr.w, j, sc, mn);
                dsc[j] = d * (float)sc;
                dmn[j] = dmin * (float)mn;
            }
            // this lane's token: activation scale and scale * sum(q) of the eight sub-blocks
            const float4 dxa = *reinterpret_cast<const float4 *>(xrow + sb * 8), dxb = *reinterpret_cast<const float4 *>(xrow + sb * 8 + 4);
            const float4 sxa = *reinterpret_cast<const float4 *>(srow + sb * 8), sxb = *reinterpret_cast<const float4 *>(srow + sb * 8 + 4);
            const float dxl[8] = {dxa.x, dxa.y, dxa.z, dxa.w, dxb.x, dxb.y, dxb.z, dxb.w};
            const float sxl[8] = {sxa.x, sxa.y, sxa.z, sxa.w, sxb.x, sxb.y, sxb.z, sxb.w};
            uint2 aq[4][4];
#pragma unroll
            for (int gq = 0; gq < 4; ++gq)
#pragma unroll
                for (int j = 0; j < 4; ++j) aq[gq][j] = ldg8(arow[j] + (size_t)sb * 144 + 32 * gq);
#pragma unroll
            for (int gq = 0; gq < 4; ++gq) {
                const uint2 (&a)[4] = aq[gq];
#pragma unroll
                for (int hi = 0; hi < 2; ++hi) {
                    const int j8 = 2 * gq + hi;  // sub-block
                    const int koff = (sb * 8 + j8) * 32;
                    uint2 b[NT];
#pragma unroll
                    for (int t = 0; t < NT; ++t) b[t] = ldg8(brow[t] + koff);
                    float ws[2][2], wm[2][2];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int src = (j >> 1) * 16 + g + (j & 1) * 8;
                        ws[j >> 1][j & 1] = __shfl_sync(0xffffffffu, dsc[j8], src);
                        wm[j >> 1][j & 1] = __shfl_sync(0xffffffffu, dmn[j8], src);
                    }
                    uint32_t an[4][2];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        an[j][0] = (hi ? (a[j].x >> 4) : a[j].x) & 0x0F0F0F0Fu;
                        an[j][1] = (hi ? (a[j].y >> 4) : a[j].y) & 0x0F0F0F0Fu;
                    }
#pragma unroll
                    for (int t = 0; t < NT; ++t) {
                        const float dx0 = __shfl_sync(0xffffffffu, dxl[j8], 8 * t + 2 * tg);
                        const float dx1 = __shfl_sync(0xffffffffu, dxl[j8], 8 * t + 2 * tg + 1);
                        const float sx0 = __shfl_sync(0xffffffffu, sxl[j8], 8 * t + 2 * tg);
                        const float sx1 = __shfl_sync(0xffffffffu, sxl[j8], 8 * t + 2 * tg + 1);
#pragma unroll
                        for (int mt = 0; mt < 2; ++mt) {
                            int c[4];
                            mma_s8(c, an[2 * mt][0], an[2 * mt + 1][0], an[2 * mt][1], an[2 * mt + 1][1], b[t].x, b[t].y);
                            acc[mt][t][0] = fmaf(-wm[mt][0], sx0, fmaf((float)c[0], ws[mt][0] * dx0, acc[mt][t][0]));
                            acc[mt][t][1] = fmaf(-wm[mt][0], sx1, fmaf((float)c[1], ws[mt][0] * dx1, acc[mt][t][1]));
                            acc[mt][t][2] = fmaf(-wm[mt][1], sx0, fmaf((float)c[2], ws[mt][1] * dx0, acc[mt][t][2]));
                            acc[mt][t][3] = fmaf(-wm[mt][1], sx1, fmaf((float)c[3], ws[mt][1] * dx1, acc[mt][t][3]));
                        }
                    }
                }
            }
        }
        reduce_and_store<NT>(red, acc, out, N, M, r0, t0);
    }
}

// ------------------------------------------------------------------------------------------------ Q6_K
// Weights in the unit layout of smc_common.cuh (X, Y, Z entries per lane slot, 16 int8 scales and fp16 d per block).
// A scale covers 16 elements, so the unit is mma.m16n8k16: for half h (128 elements) and sixteen `is` a lane reads
// four bytes of the X, Y and Z entries of slot (block, h, is) at byte 4*tg of each of its four rows and forms from
// them the codes of columns c = 0..3 (elements 32c + l .. l + 3 of the half, l = 16*is + 4*tg), 32 subtracted
// bytewise; out += (d * sc[8h + is + 2c]) * dx[4h + c] * isum.
__device__ __forceinline__ void mma_s8_k16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0)
{
    asm("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
        : "r"(a0), "r"(a1), "r"(b0), "r"(0));
}

__device__ __forceinline__ uint32_t ldg4(const void *p)
{
    uint32_t v;
    asm("ld.global.nc.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

template <int C>
__device__ __forceinline__ uint32_t q6_codes(uint32_t wx, uint32_t wy, uint32_t wz)
{
    const uint32_t M6 = 0x3F3F3F3Fu;
    uint32_t q;
    if (C == 0) q = wx & M6;
    else if (C == 1) q = wy & M6;
    else if (C == 2) q = wz & M6;
    else q = ((wx >> 6) & 0x03030303u) | ((wy >> 4) & 0x0C0C0C0Cu) | ((wz >> 2) & 0x30303030u);
    return __vsub4(q, 0x20202020u);  // codes 0..63 -> -32..31, no byte borrows into its neighbour
}

template <int NT, int NW>
__global__ void __launch_bounds__(NW * 32, NW == 8 ? 2 : 1)
gemv_mma_q6_K_kernel(const uint8_t *__restrict__ q6u, const int8_t *__restrict__ xq, const float *__restrict__ xd,
                     float *__restrict__ out, int N, int K, int M)
{
    // NW warps split K: 8 (two CTAs per SM), or 16 in one CTA per SM for rows of 8192 elements and more
    extern __shared__ __align__(16) float red_dyn[];
    float (*red)[8 * NT][RED_LD] = reinterpret_cast<float (*)[8 * NT][RED_LD]>(red_dyn);
    smc_grid_dep_sync();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, tg = lane & 3;
    const int r0 = blockIdx.x * MMA_ROWS;
    const int nb = K / 32, nsb = K / 256;
    uint32_t rblk[4];  // block indices: a tensor has fewer than 2^32 blocks of 256
#pragma unroll
    for (int j = 0; j < 4; ++j) rblk[j] = (uint32_t)min(r0 + (j >> 1) * 16 + g + (j & 1) * 8, N - 1) * (uint32_t)nsb;
    const uint32_t hblk = (uint32_t)min(r0 + lane, N - 1) * (uint32_t)nsb;
    {  // one pass of 8 * NT tokens per CTA: blockIdx.y picks the pass (a batch of more than 32 rows fills the grid with passes)
        const int t0 = blockIdx.y * 8 * NT;
        const int8_t *brow[NT];
#pragma unroll
        for (int t = 0; t < NT; ++t) brow[t] = xq + (size_t)min(t0 + 8 * t + g, M - 1) * K + 4 * tg;
        const float *xrow = xd + (size_t)min(t0 + lane, M - 1) * nb;
        float acc[2][NT][4];
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int t = 0; t < NT; ++t)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[mt][t][i] = 0.f;
        for (int sb = warp; sb < nsb; sb += NW) {
            // this lane's row: d * sc of the sixteen sub-blocks
            const uint4 scw = *reinterpret_cast<const uint4 *>(q6u + smc_q6u_scales(hblk + sb));
            const float d = __half2float(*reinterpret_cast<const __half *>(q6u + smc_q6u_d(hblk + sb)));
            // this lane's token: activation scales of the eight 32-element blocks
            const float4 dxa = *reinterpret_cast<const float4 *>(xrow + sb * 8), dxb = *reinterpret_cast<const float4 *>(xrow + sb * 8 + 4);
            // up to 16 tokens both halves are unrolled and their loads overlap; beyond, the accumulators need the registers
#pragma unroll(NT <= 2 ? 2 : 1)
            for (int h = 0; h < 2; ++h) {
                const uint32_t scws[2] = {h ? scw.z : scw.x, h ? scw.w : scw.y};
                const float dxl[4] = {h ? dxb.x : dxa.x, h ? dxb.y : dxa.y, h ? dxb.z : dxa.z, h ? dxb.w : dxa.w};
#pragma unroll
                for (int is = 0; is < 2; ++is) {
                    uint32_t wa[4], wb[4], wh[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const uint8_t *pl = q6u + smc_q6u_slot(rblk[j] + sb, h, is) + 4 * tg;
                        wa[j] = ldg4(pl), wb[j] = ldg4(pl + SMC_Q6U_Y), wh[j] = ldg4(pl + SMC_Q6U_Z);
                    }
                    auto column = [&](auto cc) {
                        constexpr int c = decltype(cc)::value;
                        constexpr int bx = c;
                        const int si = is + 2 * c;  // scale byte within the half
                        const int koff = sb * 256 + 128 * h + 32 * c + 16 * is;
                        uint32_t b[NT], an[4];
#pragma unroll
                        for (int t = 0; t < NT; ++t) b[t] = ldg4(brow[t] + koff);
#pragma unroll
                        for (int j = 0; j < 4; ++j) an[j] = q6_codes<c>(wa[j], wb[j], wh[j]);
                        const float dsc = d * (float)(int)(int8_t)((scws[si >> 2] >> (8 * (si & 3))) & 0xFF);
                        float ws[2][2];
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            ws[j >> 1][j & 1] = __shfl_sync(0xffffffffu, dsc, (j >> 1) * 16 + g + (j & 1) * 8);
#pragma unroll
                        for (int t = 0; t < NT; ++t) {
                            const float dx0 = __shfl_sync(0xffffffffu, dxl[bx], 8 * t + 2 * tg);
                            const float dx1 = __shfl_sync(0xffffffffu, dxl[bx], 8 * t + 2 * tg + 1);
#pragma unroll
                            for (int mt = 0; mt < 2; ++mt) {
                                int c4[4];
                                mma_s8_k16(c4, an[2 * mt], an[2 * mt + 1], b[t]);
                                acc[mt][t][0] = fmaf((float)c4[0], ws[mt][0] * dx0, acc[mt][t][0]);
                                acc[mt][t][1] = fmaf((float)c4[1], ws[mt][0] * dx1, acc[mt][t][1]);
                                acc[mt][t][2] = fmaf((float)c4[2], ws[mt][1] * dx0, acc[mt][t][2]);
                                acc[mt][t][3] = fmaf((float)c4[3], ws[mt][1] * dx1, acc[mt][t][3]);
                            }
                        }
                    };
                    column(std::integral_constant<int, 0>{});
                    column(std::integral_constant<int, 1>{});
                    column(std::integral_constant<int, 2>{});
                    column(std::integral_constant<int, 3>{});
                }
            }
        }
        reduce_and_store<NT, NW, 8 * NT>(red, acc, out, N, M, r0, t0);
    }
}

// ------------------------------------------------------------------------------------------ prompt sizes, Q8_0 and Q6_K
// The same sums with no split over warps: with hundreds of tokens a warp owns an output tile of 32 rows x 8 NT tokens, walks the classes of
// groups that the kernels above give to their eight (sixteen) warps one after the other, and adds each finished class to a running
// total: the same partial sums added in the same order, hence the same bits.
//
// A CTA is two row warps x two token warps: 64 rows x 16 NT tokens.  Weights, activations and scales of a group (128 elements of Q8_0, 256
// of Q6_K) come to shared memory by asynchronous copies, S groups in flight; a weight row or token takes an odd multiple of 16 bytes there,
// so that an ldmatrix of eight of them is free of conflicts.  The tokens' scales are stored so that the 2 NT of a lane lie side by side:
// a 16-byte load brings four.  Products of scales and fused multiply-adds are done two at a time (each half rounds as the scalar one).
// (The first form fetched fragments and scales from global memory and handed scales round by shuffles, which the four schedulers of an SM
// share at one per clock: Q8_0 6144 x 1024 with 2048 tokens spent 55 clocks per scheduler on an MMA and its 12 scaling operations.)
// What bounds it: 15 instructions per MMA at half the issue rate; mma.sync and the fp32 pipe exclude each other (an MMA with its conversions
// and scaling alone takes 25 clocks, the kernel 28).  The sums from tcgen05.mma kind::f16 (exact in its fp32 accumulators) were no faster:
// two drain warps per scheduler took 24 clocks per MMA's worth.
// Measured, us (before): Q8_0 6144 x 1024, 2048 tokens 155 -> 103, 4096 x 1024 105 -> 69, 1024 x 3072 67 -> 52, 1024 x 2048 48 -> 38, 4096 x 1024
// with 333 25 -> 19; Q6_K 4096 x 14336, 777 tokens 833 -> 615.
__device__ __forceinline__ uint32_t smem_at(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
template <int B>
__device__ __forceinline__ void copy_async(uint32_t dst, const void *src)
{
    if constexpr (B == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(B) : "memory");
}
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t &a, uint32_t &b, uint32_t &c, uint32_t &d)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(a), "=r"(b), "=r"(c), "=r"(d) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm2(uint32_t addr, uint32_t &a, uint32_t &b)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(a), "=r"(b) : "r"(addr) : "memory");
}
__device__ __forceinline__ uint2 lds8(uint32_t a)
{
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
    return v;
}
typedef unsigned long long f32x2;  // two floats in a register pair
__device__ __forceinline__ f32x2 pair_x2(float a, float b)
{
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpair_x2(f32x2 v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 add_x2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul_x2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma_x2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

constexpr int TILE_ROWS = 64, TILE_THREADS = 128;
template <bool Q6, int NT>
struct TileShape {
    static constexpr int TOK = 16 * NT, KG = Q6 ? 256 : 128, NB = KG / 32, S = 2;  // tokens; elements and 32-element blocks of a group; groups in flight
    static constexpr int WROW = Q6 ? 208 : 144, XROW = KG + 16;                     // bytes of a weight row (Q8_0: 128 and its four scales) and of a token
    static constexpr int DXS = NT == 8 ? 20 : NT == 6 ? 12 : 2 * NT;               // floats between the lanes' token scales: off each other's banks
    static constexpr int OFF_X = TILE_ROWS * WROW, OFF_DX = OFF_X + TOK * XROW, OFF_D = OFF_DX + 2 * NB * 4 * DXS * 4;
    static constexpr int STAGE = OFF_D + (Q6 ? TILE_ROWS * 4 : 0), SMEM = S * STAGE;
    static_assert(STAGE % 16 == 0 && NT % 2 == 0, "alignment");
};

template <bool Q6, int NT, int CTAS>
__global__ void __launch_bounds__(TILE_THREADS, CTAS)
gemv_mma_tile_kernel(const uint8_t *__restrict__ w, const __half *__restrict__ wd, const int8_t *__restrict__ xq, const float *__restrict__ xd,
                     float *__restrict__ out, int N, int K, int M, int ncls)
{
    using P = TileShape<Q6, NT>;
    extern __shared__ __align__(16) uint8_t sm_tile[];
    const uint32_t base = smem_at(sm_tile);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, tg = lane & 3, wr = warp >> 1, wt = warp & 1;
    const int r0 = blockIdx.x * TILE_ROWS, t0 = blockIdx.y * P::TOK, nb = K / 32, ngroups = K / P::KG;

    int a_cls = 0, a_gi = 0;  // the group to be requested next: classes in turn, groups cls, cls + ncls, ... of each
    auto request = [&](int slot) {
        if (a_cls < ncls && a_gi < ngroups) {
            const uint32_t st = base + (uint32_t)slot * P::STAGE;
            constexpr int PIECES = Q6 ? 13 : 8, XP = P::KG / 16;
#pragma unroll
            for (int i = 0; i < (TILE_ROWS * PIECES + TILE_THREADS - 1) / TILE_THREADS; ++i) {
                const int e = threadIdx.x + i * TILE_THREADS;
                if (TILE_ROWS * PIECES % TILE_THREADS && e >= TILE_ROWS * PIECES) break;
                const int r = e / PIECES, c = e % PIECES;
                // What lies past the last row or token is not loaded (nor stored: outputs do not mix).  Clamped to the last token, a ragged tile
                // of every CTA asked the same L2 lines for it: 6144 x 1024 Q8_0 with 300 tokens took 52 us, with 256 21.
                if (r0 + r >= N) break;
                const size_t row = (size_t)(r0 + r);
                const uint8_t *src;
                if (Q6) {
                    const size_t blk = row * ngroups + a_gi;
                    src = c < 12 ? w + smc_q6u_slot(blk, 0, 0) + 512 * (c >> 2) + 16 * (c & 3) : w + smc_q6u_scales(blk);
                } else src = w + row * K + a_gi * 128 + 16 * c;
                copy_async<16>(st + (uint32_t)(r * P::WROW + 16 * c), src);
            }
            if (threadIdx.x < TILE_ROWS && r0 + (int)threadIdx.x < N) {  // Q8_0: four scales behind the row's codes; Q6_K: the aligned four bytes that hold the block's d
                const size_t row = (size_t)(r0 + (int)threadIdx.x);
                if (Q6) copy_async<4>(st + (uint32_t)(P::OFF_D + 4 * threadIdx.x), w + (smc_q6u_d(row * ngroups + a_gi) & ~(size_t)3));
                else copy_async<8>(st + (uint32_t)(threadIdx.x * P::WROW + 128), wd + row * nb + a_gi * 4);
            }
#pragma unroll
            for (int i = 0; i < P::TOK * XP / TILE_THREADS; ++i) {
                const int e = threadIdx.x + i * TILE_THREADS, t = e / XP, c = e % XP;
                if (t0 + t < M) copy_async<16>(st + (uint32_t)(P::OFF_X + t * P::XROW + 16 * c), xq + (size_t)(t0 + t) * K + a_gi * P::KG + 16 * c);
            }
#pragma unroll
            for (int i = 0; i < P::TOK * P::NB / TILE_THREADS; ++i) {
                const int e = threadIdx.x + i * TILE_THREADS, t = e / P::NB, b = e % P::NB, u = t % (8 * NT);
                if (t0 + t < M)
                    copy_async<4>(st + (uint32_t)(P::OFF_DX + 4 * ((((t / (8 * NT)) * P::NB + b) * 4 + ((u & 7) >> 1)) * P::DXS + 2 * (u >> 3) + (u & 1))),
                                  xd + (size_t)(t0 + t) * nb + a_gi * P::NB + b);
            }
            a_gi += ncls;
            while (a_gi >= ngroups && a_cls < ncls) a_gi = ++a_cls;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    static_assert(P::TOK * (P::KG / 16) % TILE_THREADS == 0 && P::TOK * P::NB % TILE_THREADS == 0, "copies per thread");
    smc_grid_dep_sync();
#pragma unroll
    for (int i = 0; i < P::S - 1; ++i) request(i);

    // this lane's ldmatrix rows
    const uint32_t a_off = (uint32_t)((wr * 32 + (lane & 7) + 8 * ((lane >> 3) & 1)) * P::WROW + 16 * (lane >> 4));
    const uint32_t b_off = (uint32_t)(P::OFF_X + wt * 8 * NT * P::XROW), dx_off = (uint32_t)(P::OFF_DX + (wt * P::NB * 4 + tg) * P::DXS * 4);
    f32x2 acc[2][NT][2], total[2][NT][2];  // [16-row tile][token tile][rows g, g + 8]: tokens 2 tg, 2 tg + 1
    auto scale_add = [&](f32x2 (&a)[2], const int (&c)[4], const f32x2 (&ws)[2], f32x2 dx) {
        a[0] = fma_x2(pair_x2((float)c[0], (float)c[1]), mul_x2(ws[0], dx), a[0]);
        a[1] = fma_x2(pair_x2((float)c[2], (float)c[3]), mul_x2(ws[1], dx), a[1]);
    };
    auto token_scales = [&](uint32_t at, f32x2 (&v)[NT]) {
#pragma unroll
        for (int t = 0; t < NT; t += 2) asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(v[t]), "=l"(v[t + 1]) : "r"(at + 8u * t) : "memory");
    };
    auto group_q8 = [&](uint32_t st) {
        uint2 dw[2][2];
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int h = 0; h < 2; ++h) dw[mt][h] = lds8(st + (uint32_t)((wr * 32 + 16 * mt + 8 * h + g) * P::WROW + 128));
#pragma unroll
        for (int kb = 0; kb < 4; ++kb) {
            uint32_t a[2][4], b[NT][2];
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) ldsm4(st + a_off + (uint32_t)(16 * mt * P::WROW + 32 * kb), a[mt][0], a[mt][1], a[mt][2], a[mt][3]);
#pragma unroll
            for (int t = 0; t < NT; t += 2)
                ldsm4(st + b_off + (uint32_t)((8 * t + (lane & 7) + 8 * (lane >> 4)) * P::XROW + 32 * kb + 16 * ((lane >> 3) & 1)), b[t][0], b[t][1], b[t + 1][0], b[t + 1][1]);
            f32x2 dx[NT], ws[2][2];
            token_scales(st + dx_off + (uint32_t)(kb * 16 * P::DXS), dx);
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t two = (kb & 2) ? dw[mt][h].y : dw[mt][h].x;
                    const float d = smc_h2f((uint16_t)((kb & 1) ? (two >> 16) : (two & 0xFFFFu)));
                    ws[mt][h] = pair_x2(d, d);
                }
#pragma unroll
            for (int t = 0; t < NT; ++t)
#pragma unroll
                for (int mt = 0; mt < 2; ++mt) {
                    int c[4];
                    mma_s8(c, a[mt][0], a[mt][1], a[mt][2], a[mt][3], b[t][0], b[t][1]);
                    scale_add(acc[mt][t], c, ws[mt], dx[t]);
                }
        }
    };
    auto group_q6 = [&](uint32_t st, int gi) {
        float d[2][2];
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int r = wr * 32 + 16 * mt + 8 * u + g;
                uint32_t two;
                asm volatile("ld.shared.u32 %0, [%1];" : "=r"(two) : "r"(st + (uint32_t)(P::OFF_D + 4 * r)) : "memory");
                const bool odd = ((uint32_t)(r0 + r) * (uint32_t)ngroups + (uint32_t)gi) & 1u;  // of the block's number
                d[mt][u] = smc_h2f((uint16_t)(odd ? two >> 16 : two & 0xFFFFu));
            }
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
            uint2 sc[2][2];  // this half's scale bytes: is + 2 c
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int u = 0; u < 2; ++u) sc[mt][u] = lds8(st + (uint32_t)((wr * 32 + 16 * mt + 8 * u + g) * P::WROW + 192 + 8 * h));
#pragma unroll
            for (int is = 0; is < 2; ++is) {
                uint32_t X[2][2], Y[2][2], Z[2][2];  // matrix i of an ldmatrix: rows 8 i .. 8 i + 7 of the warp's 32
                const uint32_t at = st + (uint32_t)((wr * 32 + lane) * P::WROW + 32 * h + 16 * is);
                ldsm4(at, X[0][0], X[0][1], X[1][0], X[1][1]);
                ldsm4(at + 64, Y[0][0], Y[0][1], Y[1][0], Y[1][1]);
                ldsm4(at + 128, Z[0][0], Z[0][1], Z[1][0], Z[1][1]);
#pragma unroll
                for (int c4 = 0; c4 < 4; ++c4) {
                    uint32_t b[NT], a[2][2];
                    const uint32_t kh = 128u * h + 32u * c4 + 16u * is;
#pragma unroll
                    for (int t = 0; t < NT; t += 4) {
                        if (NT - t >= 4) ldsm4(st + b_off + (uint32_t)((8 * t + lane) * P::XROW) + kh, b[t], b[t + 1], b[t + 2], b[t + 3]);
                        else ldsm2(st + b_off + (uint32_t)((8 * t + (lane & 15)) * P::XROW) + kh, b[t], b[t + 1]);
                    }
                    f32x2 dx[NT], ws[2][2];
                    token_scales(st + dx_off + (uint32_t)((4 * h + c4) * 16 * P::DXS), dx);
#pragma unroll
                    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const uint32_t wx = X[mt][u], wy = Y[mt][u], wz = Z[mt][u];
                            uint32_t q;  // codes 0 .. 63, then 32 taken off bytewise: 0x80 keeps the borrow inside a byte
                            if (c4 == 0) q = wx & 0x3F3F3F3Fu;
                            else if (c4 == 1) q = wy & 0x3F3F3F3Fu;
                            else if (c4 == 2) q = wz & 0x3F3F3F3Fu;
                            else q = ((wx >> 6) & 0x03030303u) | ((wy >> 4) & 0x0C0C0C0Cu) | ((wz >> 2) & 0x30303030u);
                            a[mt][u] = ((q | 0x80808080u) - 0x20202020u) ^ 0x80808080u;
                            const int si = is + 2 * c4;
                            const uint32_t word = si < 4 ? sc[mt][u].x : sc[mt][u].y;
                            const float s = d[mt][u] * (float)(int)(int8_t)((word >> (8 * (si & 3))) & 0xFFu);
                            ws[mt][u] = pair_x2(s, s);
                        }
#pragma unroll
                    for (int t = 0; t < NT; ++t)
#pragma unroll
                        for (int mt = 0; mt < 2; ++mt) {
                            int c[4];
                            mma_s8_k16(c, a[mt][0], a[mt][1], b[t]);
                            scale_add(acc[mt][t], c, ws[mt], dx[t]);
                        }
                }
            }
        }
    };
    int slot = 0;
#pragma unroll 1
    for (int cls = 0; cls < ncls; ++cls) {
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int t = 0; t < NT; ++t) acc[mt][t][0] = acc[mt][t][1] = 0ull;
#pragma unroll 1
        for (int gi = cls; gi < ngroups; gi += ncls) {
            asm volatile("cp.async.wait_group %0;" ::"n"(P::S - 2) : "memory");
            __syncthreads();  // the group has landed for everybody, and everybody is through with the slot that is refilled
            request(slot == 0 ? P::S - 1 : slot - 1);
            const uint32_t st = base + (uint32_t)slot * P::STAGE;
            if constexpr (Q6) group_q6(st, gi);
            else group_q8(st);
            if (++slot == P::S) slot = 0;
        }
        // the split kernels' fold: s = partial of warp 0; s += partial of warp 1; ...
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int t = 0; t < NT; ++t)
#pragma unroll
                for (int h = 0; h < 2; ++h) total[mt][t][h] = cls == 0 ? acc[mt][t][h] : add_x2(total[mt][t][h], acc[mt][t][h]);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float v[2];
                unpair_x2(total[mt][t][h], v[0], v[1]);
                const int row = r0 + wr * 32 + 16 * mt + 8 * h + g, tok = t0 + wt * 8 * NT + 8 * t + 2 * tg;
                if (row < N && tok < M) out[(size_t)tok * N + row] = v[0];
                if (row < N && tok + 1 < M) out[(size_t)(tok + 1) * N + row] = v[1];
            }
}

// ------------------------------------------------------------------------------------------ 2 .. 63 rows, Q8_0 and Q4_K, staged
// The same sums again, for batches that the tiles above are too large for.  A CTA takes jobs of 32 WR weight rows x 8 NT tokens; its 8 / WR groups of WR warps
// take the classes of K groups as the warps of the split kernels do (a group of fewer than eight takes several, one after the other)
// and meet in shared memory, where each output is added up in class order: the same bits.  Each group of warps has its own ring of S stages (a
// stage: a class's next 128 elements of Q8_0 or 256 of Q4_K, of all rows and tokens of the job), filled by asynchronous copies, and with one warp to a
// group it waits for nobody else's.  A CTA is one per SM and goes from job to job with its copies running ahead; the first weights are asked
// for before the predecessor is waited for.  Layout in a stage, scales and products are the tile kernel's.  Q4_K: a warp writes its rows'
// d * sc and dmin * m of a 256-block to a table once, instead of handing them round by shuffles.
// What bounds it: the MMAs with their scaling are 24 of 57 us (Q4_K 28672 x 4096, 32 rows, 25 - 30 clocks each) and 6 of 29 with 6 rows, the weights' bytes 10; the
// rest is a warp's own chain of copy, wait, fragments and sums, with one or two steps in flight and eight warps to an SM.
// The split kernels that ran here had their fragments as 8-byte loads from global memory, just in time, and 8 shuffles per MMA's tokens.
// Measured, us (before): Q4_K 28672 x 4096 with 6 rows 33.5 -> 28.8, 16 45.2 -> 40.5, 32 70.9 -> 57.5; 4096 x 14336, 6 20.5 -> 14.5; 6144 x 4096, 32
// 22.7 -> 18.6; 1024 x 4096, 32 12.4 -> 6.5; Q8_0 1024 x 3072, 32 10.4 -> 6.1; 4096 x 14336, 6 24.7 -> 16.5, 16 27.1 -> 20.7, 32 37.1 -> 25.3; 6144 x
// 1024, 32 8.7 -> 8.3.
template <bool Q4, int WR, int NT, int S>
struct StageShape {
    static constexpr int WK = MMA_WARPS / WR, GROUP = 32 * WR;
    static constexpr int ROWS = 32 * WR, TOK = 8 * NT, KG = Q4 ? 256 : 128, NB = KG / 32;
    static constexpr int WROW = 144, XROW = KG + 16, DXS = 2 * NT;  // Q8_0: 128 codes and their four scales; Q4_K: a block
    static constexpr int DXB = NB * 4 * DXS * 4;
    static constexpr int OFF_X = ROWS * WROW, OFF_DX = OFF_X + TOK * XROW, OFF_SX = OFF_DX + DXB, STAGE = OFF_SX + (Q4 ? DXB : 0);
    static constexpr int TAB = Q4 ? 32 * 80 : 0;  // a warp's rows' eight (d sc, dmin m), 64 bytes on 80
    static constexpr int OFF_TAB = WK * S * STAGE, OFF_RED = OFF_TAB + MMA_WARPS * TAB;
    static constexpr int RLD = ROWS + 4, RED = WK * TOK * RLD * 4;
    static constexpr int REDS = OFF_RED + 2 * RED <= 227 * 1024 ? 2 : 1;  // two: the next round's partial sums need not wait for this one's readers
    static constexpr int SMEM = OFF_RED + REDS * RED;
    static_assert(STAGE % 16 == 0 && OFF_TAB % 16 == 0 && SMEM <= 227 * 1024, "shared memory");
};

template <bool Q4, int WR, int NT, int S>
__global__ void __launch_bounds__(32 * MMA_WARPS, 1)
gemv_mma_staged_kernel(const uint8_t *__restrict__ w, const __half *__restrict__ wd, const int8_t *__restrict__ xq, const float *__restrict__ xd,
                       const float *__restrict__ xsd, float *__restrict__ out, int N, int K, int M, int passes, int jobs)
{
    using P = StageShape<Q4, WR, NT, S>;
    constexpr int WK = P::WK;
    extern __shared__ __align__(16) uint8_t sm_staged[];
    const uint32_t base = smem_at(sm_staged);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, tg = lane & 3;
    const int wk = warp / WR, wr = warp % WR, gt = threadIdx.x % P::GROUP;
    const int nb = K / 32, ngroups = K / P::KG;
    const uint32_t ring = base + (uint32_t)(wk * S) * P::STAGE;

    // the step whose bytes are asked for next: job, class, K group
    int a_job = blockIdx.x, a_cls = wk, a_gi = wk;
    auto settle = [&]() {  // over classes that have no (more) steps
        while (a_job < jobs && a_gi >= ngroups) {
            a_cls += WK;
            if (a_cls >= MMA_WARPS) a_cls = wk, a_job += gridDim.x;
            a_gi = a_cls;
            if (wk >= ngroups) a_job = jobs;  // none of this group's classes has any
        }
    };
    // What lies past the last row or token is not loaded (nor stored: outputs do not mix).
    auto request_weights = [&](int slot) {
        const uint32_t st = ring + (uint32_t)slot * P::STAGE;
        const int r0 = a_job / passes * P::ROWS;
        constexpr int PIECES = Q4 ? 9 : 8;
#pragma unroll
        for (int i = 0; i < P::ROWS * PIECES / P::GROUP; ++i) {
            const int e = gt + i * P::GROUP, r = e / PIECES, c = e % PIECES;
            if (r0 + r >= N) break;
            const size_t row = (size_t)(r0 + r);
            copy_async<16>(st + (uint32_t)(r * P::WROW + 16 * c), Q4 ? w + (row * ngroups + a_gi) * 144 + 16 * c : w + row * K + a_gi * 128 + 16 * c);
        }
        if (!Q4 && r0 + gt < N) copy_async<8>(st + (uint32_t)(gt * P::WROW + 128), wd + (size_t)(r0 + gt) * nb + a_gi * 4);
    };
    auto request_tokens = [&](int slot) {
        const uint32_t st = ring + (uint32_t)slot * P::STAGE;
        const int t0 = a_job % passes * P::TOK;
        constexpr int XP = P::KG / 16;
#pragma unroll
        for (int i = 0; i < P::TOK * XP / P::GROUP; ++i) {
            const int e = gt + i * P::GROUP, t = e / XP, c = e % XP;
            if (t0 + t < M) copy_async<16>(st + (uint32_t)(P::OFF_X + t * P::XROW + 16 * c), xq + (size_t)(t0 + t) * K + a_gi * P::KG + 16 * c);
        }
#pragma unroll
        for (int i = 0; i < (P::TOK * P::NB + P::GROUP - 1) / P::GROUP; ++i) {
            const int e = gt + i * P::GROUP, t = e / P::NB, b = e % P::NB;
            if (t < P::TOK && t0 + t < M) {
                const uint32_t at = 4u * (uint32_t)((b * 4 + ((t & 7) >> 1)) * P::DXS + 2 * (t >> 3) + (t & 1));
                const size_t from = (size_t)(t0 + t) * nb + a_gi * P::NB + b;
                copy_async<4>(st + P::OFF_DX + at, xd + from);
                if (Q4) copy_async<4>(st + P::OFF_SX + at, xsd + from);
            }
        }
    };
    auto advance = [&]() { a_gi += MMA_WARPS, settle(); };
    static_assert(P::ROWS == P::GROUP && P::ROWS * (Q4 ? 9 : 8) % P::GROUP == 0 && P::TOK * (P::KG / 16) % P::GROUP == 0, "copies per thread");

    settle();
    const int f_job = a_job, f_cls = a_cls, f_gi = a_gi;
#pragma unroll
    for (int i = 0; i < S - 1; ++i)
        if (a_job < jobs) request_weights(i), advance();
    a_job = f_job, a_cls = f_cls, a_gi = f_gi;
    smc_grid_dep_sync();
#pragma unroll
    for (int i = 0; i < S - 1; ++i) {  // (the first of these groups holds all the weights)
        if (a_job < jobs) request_tokens(i), advance();
        asm volatile("cp.async.commit_group;" ::: "memory");
    }

    // this lane's ldmatrix rows
    const uint32_t a_off = (uint32_t)((wr * 32 + (lane & 7) + 8 * ((lane >> 3) & 1)) * P::WROW + 16 * (lane >> 4));
    const uint32_t dx_off = (uint32_t)(P::OFF_DX + tg * P::DXS * 4);
    const uint32_t tab = base + P::OFF_TAB + (uint32_t)warp * P::TAB;
    f32x2 acc[2][NT][2];  // [16-row tile][token tile][rows g, g + 8]: tokens 2 tg, 2 tg + 1
    auto scale_add = [&](f32x2 (&a)[2], const int (&c)[4], const f32x2 (&ws)[2], f32x2 dx) {
        a[0] = fma_x2(pair_x2((float)c[0], (float)c[1]), mul_x2(ws[0], dx), a[0]);
        a[1] = fma_x2(pair_x2((float)c[2], (float)c[3]), mul_x2(ws[1], dx), a[1]);
    };
    auto token_scales = [&](uint32_t at, f32x2 (&v)[NT]) {
        if constexpr (NT == 1) asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v[0]) : "r"(at) : "memory");
        else {
#pragma unroll
            for (int t = 0; t < NT; t += 2) asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(v[t]), "=l"(v[t + 1]) : "r"(at + 8u * t) : "memory");
        }
    };
    auto token_codes = [&](uint32_t st, int k, uint32_t (&b)[NT][2]) {  // of the 32-element block at byte k of the stage's token rows
        const uint32_t at = st + P::OFF_X + (uint32_t)((lane & 7) * P::XROW + k + 16 * ((lane >> 3) & 1));
        if constexpr (NT == 1) ldsm2(at, b[0][0], b[0][1]);
        else {
#pragma unroll
            for (int t = 0; t < NT; t += 2) ldsm4(at + (uint32_t)((8 * t + 8 * (lane >> 4)) * P::XROW), b[t][0], b[t][1], b[t + 1][0], b[t + 1][1]);
        }
    };
    auto step_q8 = [&](uint32_t st) {
        uint2 dw[2][2];
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int h = 0; h < 2; ++h) dw[mt][h] = lds8(st + (uint32_t)((wr * 32 + 16 * mt + 8 * h + g) * P::WROW + 128));
#pragma unroll
        for (int kb = 0; kb < 4; ++kb) {
            uint32_t a[2][4], b[NT][2];
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) ldsm4(st + a_off + (uint32_t)(16 * mt * P::WROW + 32 * kb), a[mt][0], a[mt][1], a[mt][2], a[mt][3]);
            token_codes(st, 32 * kb, b);
            f32x2 dx[NT], ws[2][2];
            token_scales(st + dx_off + (uint32_t)(kb * 16 * P::DXS), dx);
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t two = (kb & 2) ? dw[mt][h].y : dw[mt][h].x;
                    const float d = smc_h2f((uint16_t)((kb & 1) ? (two >> 16) : (two & 0xFFFFu)));
                    ws[mt][h] = pair_x2(d, d);
                }
#pragma unroll
            for (int t = 0; t < NT; ++t)
#pragma unroll
                for (int mt = 0; mt < 2; ++mt) {
                    int c[4];
                    mma_s8(c, a[mt][0], a[mt][1], a[mt][2], a[mt][3], b[t][0], b[t][1]);
                    scale_add(acc[mt][t], c, ws[mt], dx[t]);
                }
        }
    };
    auto step_q4 = [&](uint32_t st) {
        {
            uint4 hdr;
            asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(hdr.x), "=r"(hdr.y), "=r"(hdr.z), "=r"(hdr.w) : "r"(st + (uint32_t)((wr * 32 + lane) * P::WROW)) : "memory");
            const float d = smc_h2f((uint16_t)(hdr.x & 0xFFFFu)), dmin = smc_h2f((uint16_t)(hdr.x >> 16));
            __syncwarp();  // the previous step's table has been read
#pragma unroll
            for (int i = 0; i < 8; i += 2) {
                int s0, m0, s1, m1;
                smc_k4_scale_min(hdr.y, hdr.z, hdr.w, i, s0, m0), smc_k4_scale_min(hdr.y, hdr.z, hdr.w, i + 1, s1, m1);
                asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(tab + (uint32_t)(lane * 80 + 8 * i)), "f"(d * (float)s0), "f"(dmin * (float)m0), "f"(d * (float)s1),
                             "f"(dmin * (float)m1)
                             : "memory");
            }
            __syncwarp();
        }
#pragma unroll
        for (int gq = 0; gq < 4; ++gq) {
            uint32_t raw[2][4];
            float4 sm[2][2];
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) {
                ldsm4(st + a_off + (uint32_t)(16 * mt * P::WROW + 16 + 32 * gq), raw[mt][0], raw[mt][1], raw[mt][2], raw[mt][3]);
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];"
                                 : "=f"(sm[mt][h].x), "=f"(sm[mt][h].y), "=f"(sm[mt][h].z), "=f"(sm[mt][h].w)
                                 : "r"(tab + (uint32_t)((16 * mt + 8 * h + g) * 80 + 16 * gq))
                                 : "memory");
            }
#pragma unroll
            for (int hi = 0; hi < 2; ++hi) {
                const int j = 2 * gq + hi;  // sub-block
                uint32_t b[NT][2];
                token_codes(st, 32 * j, b);
                f32x2 dx[NT], sx[NT], ws[2][2], wm[2][2];
                token_scales(st + dx_off + (uint32_t)(j * 16 * P::DXS), dx);
                token_scales(st + dx_off + (uint32_t)(P::DXB + j * 16 * P::DXS), sx);
#pragma unroll
                for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const float s = hi ? sm[mt][h].z : sm[mt][h].x, m = -(hi ? sm[mt][h].w : sm[mt][h].y);
                        ws[mt][h] = pair_x2(s, s), wm[mt][h] = pair_x2(m, m);
                    }
#pragma unroll
                for (int t = 0; t < NT; ++t)
#pragma unroll
                    for (int mt = 0; mt < 2; ++mt) {
                        uint32_t a[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) a[i] = (hi ? raw[mt][i] >> 4 : raw[mt][i]) & 0x0F0F0F0Fu;
                        int c[4];
                        mma_s8(c, a[0], a[1], a[2], a[3], b[t][0], b[t][1]);
                        scale_add(acc[mt][t], c, ws[mt], dx[t]);
                        acc[mt][t][0] = fma_x2(wm[mt][0], sx[t], acc[mt][t][0]), acc[mt][t][1] = fma_x2(wm[mt][1], sx[t], acc[mt][t][1]);
                    }
            }
        }
    };

    constexpr int OWN = P::ROWS * P::TOK / (32 * MMA_WARPS);  // outputs of a thread
    static_assert(OWN * 32 * MMA_WARPS == P::ROWS * P::TOK, "outputs per thread");
    int slot = 0, round = 0;
#pragma unroll 1
    for (int job = blockIdx.x; job < jobs; job += gridDim.x) {
        float own[OWN];
#pragma unroll 1
        for (int cls = wk; cls < MMA_WARPS; cls += WK) {
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int t = 0; t < NT; ++t) acc[mt][t][0] = acc[mt][t][1] = 0ull;
#pragma unroll 1
            for (int gi = cls; gi < ngroups; gi += MMA_WARPS) {
                asm volatile("cp.async.wait_group %0;" ::"n"(S - 2) : "memory");
                // the step has landed for the whole group of warps, and all of it is through with the slot that is refilled
                if constexpr (WR == 1) __syncwarp();
                else asm volatile("bar.sync %0, %1;" ::"r"(1 + wk), "n"(P::GROUP) : "memory");
                if (a_job < jobs) {
                    const int next = slot == 0 ? S - 1 : slot - 1;
                    request_weights(next), request_tokens(next), advance();
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
                const uint32_t st = ring + (uint32_t)slot * P::STAGE;
                if constexpr (Q4) step_q4(st);
                else step_q8(st);
                if (++slot == S) slot = 0;
            }
            float *red = reinterpret_cast<float *>(sm_staged + P::OFF_RED + (P::REDS == 2 ? (round & 1) * P::RED : 0));
            if (P::REDS == 1 && round) __syncthreads();
            ++round;
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int t = 0; t < NT; ++t)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        float *at = red + (wk * P::TOK + 8 * t + 2 * tg) * P::RLD + wr * 32 + 16 * mt + 8 * h + g;
                        unpair_x2(acc[mt][t][h], at[0], at[P::RLD]);
                    }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < OWN; ++i) {
                const int e = threadIdx.x + i * 32 * MMA_WARPS, row = e % P::ROWS, tok = e / P::ROWS;
                float s = cls == wk ? red[tok * P::RLD + row] : own[i] + red[tok * P::RLD + row];
#pragma unroll
                for (int c = 1; c < WK; ++c) s += red[(c * P::TOK + tok) * P::RLD + row];
                own[i] = s;
            }
        }
        const int r0 = job / passes * P::ROWS, t0 = job % passes * P::TOK;
#pragma unroll
        for (int i = 0; i < OWN; ++i) {
            const int e = threadIdx.x + i * 32 * MMA_WARPS, row = r0 + e % P::ROWS, tok = t0 + e / P::ROWS;
            if (row < N && tok < M) out[(size_t)tok * N + row] = own[i];
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

}  // namespace

bool smc_mma_supported(const smc_weight *w, int M)
{
    if (!w->fast || M < 2) return false;
    if (w->dtype == SMC_Q8_0) return w->K % 128 == 0 && w->q8_qs != nullptr;
    if (w->dtype == SMC_Q4_K) return w->K % 256 == 0 && w->d_raw != nullptr;
    if (w->dtype == SMC_Q6_K) return w->K % 256 == 0 && w->q6u != nullptr;
    return false;
}

// Tokens per tile / 16 of the prompt-sized kernel for a call, 0: the kernels that split K over warps are the faster ones.
// Both run in rounds: a CTA of a kernel takes so many us per 1024 elements of K, more if others share its SM.  Measured at K = 1024 .. 28672,
// for one, two (and three) tiles on an SM; a CTA of the split kernels 2.7, and 1.8 whatever K of Q8_0 (its fold).  The estimates are within
// a tenth of these measurements (us, split kernel -> the tile chosen): Q8_0 6144 x 1024, 64 tokens 12.5 -> 10.5, 400 48 -> 29, 700 72 -> 41; 1024 x
// 3072, 256 14.3 (tiles 22.8), 512 24.5 -> 22.8, 1200 54 -> 43; Q6_K 4096 x 14336, 160 195 (213), 300 342 -> 312, 777 834 -> 615; 1024 x 4096, 600
// 58 (64), 1200 101 -> 95.
static int prompt_tile(const smc_ctx *ctx, const smc_weight *w, int M)
{
    const bool q6 = w->dtype == SMC_Q6_K;
    if (M < 64 || (w->dtype != SMC_Q8_0 && !q6)) return 0;
    const long long sms = ctx->sm_count, k = w->K;
    auto per_sm = [&](long long ctas) { return (ctas + sms - 1) / sms; };
    const long long strips = (w->N + MMA_ROWS - 1) / MMA_ROWS;
    double best = q6 ? per_sm(strips * ((M + 31) / 32)) * 2.7 * k : per_sm(strips * ((M + 63) / 64)) * (1.8 * 1024 + 2.75 * k);
    int nt = 0;
    auto offer = [&](int n, int fit, const double (&us)[3]) {  // `fit` tiles share an SM
        const long long c = per_sm(((long long)w->N + TILE_ROWS - 1) / TILE_ROWS * ((M + 16 * n - 1) / (16 * n)));
        const double t = ((c / fit) * us[fit - 1] + (c % fit ? us[c % fit - 1] : 0.0)) * k;
        if (t < best) best = t, nt = n;
    };
    if (q6) offer(4, 2, {12.6, 17.4, 0.0}), offer(6, 2, {15.2, 22.0, 0.0});
    else offer(4, 3, {6.25, 10.0, 13.75}), offer(6, 2, {8.3, 13.0, 0.0}), offer(8, 2, {10.0, 15.8, 0.0});
    return nt;
}

// The form of the staged kernel for a call; wr = 0: the Q4_K kernel that splits K over warps.
// A CTA per SM takes its jobs in rounds, each so many us per 1024 elements of K (and some 4 us a launch, the same for all): measured with one job per SM and
// with many at K = 1024 .. 28672 and 2 .. 63 rows, where the choice by these rates was never slower than the kernels it replaces.  Up to 8 tokens there is the one
// form; 9 .. 16 in one tile or two; more in tiles of 8, 16 or 32.  Narrow tiles win where weight rows are few (Q8_0 1024 x 3072, 32 tokens: 6.1 us in
// tiles of 8, 8.3 of 32; 4096 x 14336: 48 and 25).  Q4_K at 32 tokens has no room for 32 rows' rings: 64 or 128 rows to a CTA pay where they come out
// even (us, split kernel / 64 / 128 rows: 28672 x 4096 70.9 / 61.7 / 57.5, 6144 x 4096 22.7 / 18.6 / 30, 4096 x 4096 14.2 / 18.6 / 30).
struct StagedForm {
    int wr, nt;
};
static StagedForm staged_form(const smc_ctx *ctx, const smc_weight *w, int M)
{
    const bool q4 = w->dtype == SMC_Q4_K;
    double best = 1e30;
    StagedForm form{0, 0};
    auto offer = [&](int wr, int nt, double us) {
        const long long jobs = (long long)((w->N + 32 * (wr ? wr : 1) - 1) / (32 * (wr ? wr : 1))) * ((M + 8 * nt - 1) / (8 * nt));
        const double t = (double)((jobs + ctx->sm_count - 1) / ctx->sm_count) * us;
        if (t < best) best = t, form = {wr, wr ? nt : 0};
    };
    if (M > 16) q4 ? (offer(0, 4, 2.0), offer(4, 4, 6.6), offer(2, 4, 3.6)) : offer(1, 4, 1.5);
    if (M > 8) offer(1, 2, 1.2);
    offer(1, 1, q4 ? 0.75 : 0.85);
    return form;
}

// The split kernels live on L1: a lane's words are pieces of lines that its neighbours ask for.  An SM that a kernel with a large ring has left keeps its division
// into L1 and shared memory unless the next kernel asks for another, so these ask for no more shared memory than their CTAs take.  With the
// staged kernel around them and without this, a Q4_K / Q6_K decoder of 32 layers took 4322 us for 6 rows and 6376 for 32 (3547 and 5257 with it; before the staged kernel
// 4160 and 5921).  The same request from the kernels between the matmuls cost 6 % of the 6 rows.
template <class Kernel>
static void keep_l1(Kernel kernel, size_t smem, int ctas)
{
    cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, smc_l1_carveout(smem, ctas));
}

template <bool Q4, int WR, int NT, int S>
static void launch_staged(smc_ctx *ctx, const smc_q8act *a, const smc_weight *w, float *out, cudaStream_t s)
{
    using P = StageShape<Q4, WR, NT, S>;
    const auto kernel = gemv_mma_staged_kernel<Q4, WR, NT, S>;
    const int passes = (a->M + P::TOK - 1) / P::TOK, jobs = (w->N + P::ROWS - 1) / P::ROWS * passes;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, P::SMEM);
    smc_launch_dep(ctx->use_pdl, kernel, dim3(jobs < ctx->sm_count ? jobs : ctx->sm_count), dim3(32 * MMA_WARPS), P::SMEM, s,
                   Q4 ? (const uint8_t *)w->d_raw : (const uint8_t *)w->q8_qs, (const __half *)w->q8_d, (const int8_t *)a->q, (const float *)a->d, (const float *)a->sd, out,
                   w->N, w->K, a->M, passes, jobs);
}

int smc_launch_gemv_mma(smc_ctx *ctx, const smc_q8act *a, const smc_weight *w, float *out, cudaStream_t s)
{
    const int N = w->N, K = w->K, M = a->M;
    const int nt = M <= 8 ? 1 : (M <= 16 ? 2 : 4);
    const dim3 grid((N + MMA_ROWS - 1) / MMA_ROWS, (M + 8 * nt - 1) / (8 * nt));
    if (const int pt = prompt_tile(ctx, w, M)) {
        // `fit` CTAs share an SM.  A grid of fewer asks for so much shared memory that they cannot: while the kernel before it drains, the first SMs to be free
        // were given several and others none.  Measured, us (one CTA an SM): fp32 rows over Q6_K 4096 x 14336 with 63 rows (128 CTAs) 315 -> 217, Q8_0 3072 x 1024 with 50
        // (144 CTAs) 17.2 -> 13.4.
        auto go = [&](auto kernel, size_t need, int fit, int ncls) {
            const long long sms = ctx->sm_count, each = ((long long)((N + TILE_ROWS - 1) / TILE_ROWS) * ((M + 16 * pt - 1) / (16 * pt)) + sms - 1) / sms;
            const size_t alone = 228 * 1024 / 2, apart = each < fit ? 228 * 1024 / (size_t)(each + 1) : 0, smem = need > apart ? need : apart;
            cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)alone);
            const int tok = 16 * pt, most = 65535 * tok;  // tokens of a launch: what the grid's y takes
            for (int t0 = 0; t0 < M; t0 += most) {
                const int m = M - t0 < most ? M - t0 : most;
                smc_launch_dep(ctx->use_pdl, kernel, dim3((N + TILE_ROWS - 1) / TILE_ROWS, (m + tok - 1) / tok), dim3(TILE_THREADS), smem, s,
                               w->dtype == SMC_Q6_K ? (const uint8_t *)w->q6u : (const uint8_t *)w->q8_qs, (const __half *)w->q8_d, (const int8_t *)a->q + (size_t)t0 * K,
                               (const float *)a->d + (size_t)t0 * (K / 32), out + (size_t)t0 * N, N, K, m, ncls);
            }
        };
        if (w->dtype == SMC_Q6_K) {
            const int ncls = K >= 8192 ? 16 : 8;
            pt == 6 ? go(gemv_mma_tile_kernel<true, 6, 2>, TileShape<true, 6>::SMEM, 2, ncls) : go(gemv_mma_tile_kernel<true, 4, 2>, TileShape<true, 4>::SMEM, 2, ncls);
        } else if (pt == 8) go(gemv_mma_tile_kernel<false, 8, 2>, TileShape<false, 8>::SMEM, 2, 8);
        else pt == 6 ? go(gemv_mma_tile_kernel<false, 6, 2>, TileShape<false, 6>::SMEM, 2, 8) : go(gemv_mma_tile_kernel<false, 4, 3>, TileShape<false, 4>::SMEM, 3, 8);
    } else if (w->dtype == SMC_Q8_0 && M >= 64) {
        const size_t smem = (size_t)MMA_WARPS * Q8_PASS * RED_LD * sizeof(float);
        cudaFuncSetAttribute(gemv_mma_q8_0_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        keep_l1(gemv_mma_q8_0_kernel, smem, 1);
        smc_launch_dep(ctx->use_pdl, gemv_mma_q8_0_kernel, dim3((N + MMA_ROWS - 1) / MMA_ROWS, (M + Q8_PASS - 1) / Q8_PASS), dim3(256), smem, s, (const int8_t *)w->q8_qs,
                       (const __half *)w->q8_d, (const int8_t *)a->q, (const float *)a->d, out, N, K, M);
    } else if (w->dtype == SMC_Q8_0) {
        const StagedForm f = staged_form(ctx, w, M);
        f.nt == 1 ? launch_staged<false, 1, 1, 3>(ctx, a, w, out, s)
                  : f.nt == 2 ? launch_staged<false, 1, 2, 2>(ctx, a, w, out, s) : launch_staged<false, 1, 4, 2>(ctx, a, w, out, s);
    } else if (w->dtype == SMC_Q6_K) {
        // the warp count follows from K alone, so a row's bits depend neither on the batch nor on how the rows are
        // split across GPUs; long rows are where matrices of few rows (FFN down) need the extra warps per SM
        const bool wide = K >= 8192;
        auto go = [&](auto kernel, int nw) {
            const size_t smem = (size_t)nw * 8 * nt * RED_LD * sizeof(float);
            cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            keep_l1(kernel, smem, nw == 8 ? 2 : 1);
            smc_launch_dep(ctx->use_pdl, kernel, grid, dim3(nw * 32), smem, s, (const uint8_t *)w->q6u, (const int8_t *)a->q,
                           (const float *)a->d, out, N, K, M);
        };
        if (wide) {
            if (nt == 1) go(gemv_mma_q6_K_kernel<1, 16>, 16);
            else if (nt == 2) go(gemv_mma_q6_K_kernel<2, 16>, 16);
            else go(gemv_mma_q6_K_kernel<4, 16>, 16);
        } else {
            if (nt == 1) go(gemv_mma_q6_K_kernel<1, 8>, 8);
            else if (nt == 2) go(gemv_mma_q6_K_kernel<2, 8>, 8);
            else go(gemv_mma_q6_K_kernel<4, 8>, 8);
        }
    } else {
        const StagedForm f = staged_form(ctx, w, M);
        if (f.wr == 0) keep_l1(gemv_mma_q4_K_kernel, sizeof(float) * MMA_WARPS * 32 * RED_LD, 1), smc_launch_dep(ctx->use_pdl, gemv_mma_q4_K_kernel, grid, dim3(256), 0, s, (const uint8_t *)w->d_raw, (const int8_t *)a->q, (const float *)a->d,
                                      (const float *)a->sd, out, N, K, M);
        else if (f.wr == 4) launch_staged<true, 4, 4, 2>(ctx, a, w, out, s);
        else if (f.wr == 2) launch_staged<true, 2, 4, 2>(ctx, a, w, out, s);
        else f.nt == 2 ? launch_staged<true, 1, 2, 2>(ctx, a, w, out, s) : launch_staged<true, 1, 1, 3>(ctx, a, w, out, s);
    }
    SMC_LAUNCH_CHECK(ctx);
    return SMC_OK;
}
