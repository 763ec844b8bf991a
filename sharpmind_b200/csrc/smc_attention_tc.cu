// Causal prompt attention on the fifth-generation tensor cores (tcgen05 + TMEM): the arithmetic of sdpa_prefill_mma_kernel
// (smc_attention_mma.cu), which stays for short prompts, on operands split three ways, x = hi + mid + lo with every part a
// bfloat16, six products per contraction step, smallest first.
//
// tcgen05.mma kind::f16 with fp32 accumulators gives the bits of mma.sync.m16n8k16 over the same chain of K = 16 steps (compared
// over chains of up to 24 steps of mixed magnitudes), and nothing else of the order of sums changes here: scores from two
// accumulators (even and odd steps of the head size), keys in tiles of 32, running maximum, correction and row sum per tile,
// the lanes' partial row sums in the shuffle's order.  So an output has the bits it has in the other kernel, where the values that its row's last
// key tile covers are finite (below).
//
// attn_planes_kernel first writes the three planes of all keys and values a call sees, in the tensor cores' core-matrix order, V
// transposed, to scratch of the model or cache object: once per KV head instead of once per query head and row tile (split inside the attention kernel,
// by eight more warps, 2048 rows of 16 heads took 214 us, over a Q8_0 cache 281).
//
// One CTA = 128 query rows of one head; keys in chunks of 64, two tiles of 32.  Warp roles:
//   warps 0 .. 7    softmax, a thread per query row (= TMEM lane): warps 0 .. 3 the first tile of every chunk, 4 .. 7 the second.
//                   Scores out of TMEM, weights split and back into TMEM as the A operand of the second product; O (in TMEM) is
//                   multiplied by the correction unless all of a warp's are 1.  The two threads of a row exchange the tiles'
//                   maxima, corrections and row sums, so each knows the running maximum and l
//   warp 8          streams the chunks' planes by bulk copies
//   warp 9          issues the MMAs: S of the next chunk before O += P V of this one, so that they run under its softmax; the second
//                   tile's threads take their scores of that next chunk before they wait for their turn at O
// TMEM (512 columns at head size 128): Q 3 x 64, O 128, scores 2 accumulators x 64, P 3 x 16.  An MMA with the A operand in TMEM
// takes 56 clocks for any N up to 112 (64 at 128): 64 keys at once halve what the scores cost with 32.
// A row's slice of 16 leaves (O / l is stored) after the last tile that its causal bound reaches, as in the other kernel: keys of later tiles never
// meet it.  Masked keys inside that last tile enter with weight 0, so an infinite or undefined value there makes the row undefined, in both
// kernels; the other one takes keys past its CTA's 64 rows for zeros, this one those past the whole call.
// What bounds it: the softmax threads (exponentials and splits) and the order S, P, O of the chunks, which keeps the MMAs from overlapping them.
// Measured, us a call (sdpa_prefill_mma_kernel before): 2048 rows, 16 heads of 128 on 8 KV heads 362 -> 164 (Q8_0 cache 412 -> 158),
// 777 rows of 32 heads 140 -> 85, 128 rows behind 1000 keys 206 -> 90, 512 rows of heads of 64 57 -> 33.
#include <cuda_bf16.h>

#include "smc_common.cuh"
#include "smc_tc.cuh"

namespace {

constexpr size_t ATTN_PLANES_MOST = 256u << 20;  // of an object: 12 bytes an element of K, 21 000 positions of eight heads of 128; longer calls run on mma.sync
constexpr int ROWS = 128, KT = 32, CHUNK = 2 * KT, STAGES = 2;
constexpr int WARP_LOAD = 8, WARP_MMA = 9, THREADS = 32 * (WARP_MMA + 1);

template <int HD>
struct Shape {
    static constexpr uint32_t K_PLANE = CHUNK * HD * 2, V_PLANE = KT * HD * 2, V_TILE = 3 * V_PLANE;
    static constexpr uint32_t OFF_V = 3 * K_PLANE, STAGE = OFF_V + 2 * V_TILE;
    // the softmax threads' exchange: tile maxima [tile of the chunk][row], (correction, row sum) [tile][chunk parity][row]
    static constexpr uint32_t OFF_TM = STAGES * STAGE, OFF_CP = OFF_TM + 2 * ROWS * 4, OFF_BAR = OFF_CP + 4 * ROWS * 8, SMEM = OFF_BAR + 512;
    static constexpr uint32_t COL_Q = 0, Q_PLANE = HD / 2, COL_O = 3 * Q_PLANE, COL_S = COL_O + HD, COL_P = COL_S + 2 * CHUNK;
    static constexpr uint32_t COLS = 512;
    static_assert(COL_P + 3 * KT / 2 <= COLS, "tensor memory");
};
// A wait names a phase by its parity, so every barrier here is waited on by one party, phase by phase, and no phase can pass before
// that party has seen the one before it.
enum { FULL_K = 0, EMPTY_K = FULL_K + STAGES, FULL_V = EMPTY_K + STAGES, EMPTY_V = FULL_V + STAGES, S_FULL = EMPTY_V + STAGES, S_FREE, P_FULL, PV_DONE,  // PV_DONE: [tile of the chunk]
       Q_FULL = PV_DONE + 2, TM_FULL, CP_FULL = TM_FULL + 8, BARS = CP_FULL + 16 };  // TM: [tile of the chunk][warp], CP: [tile][chunk parity][warp]
static_assert(BARS * 8 + 8 <= 512, "barrier area");

__device__ __forceinline__ void mma_ta(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate)  // A in tensor memory
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
        "r"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// K-major tile without swizzle: core matrices of 8 rows x 16 bytes, lbo between neighbours along K, sbo between groups of 8 rows
__device__ __forceinline__ uint64_t desc(uint32_t addr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) | (1ull << 46);
}
__device__ __forceinline__ void st16(uint32_t taddr, const uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
        "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// two values as three bfloat16 pairs, a in the low halves (round to nearest; the remainders are exact in fp32)
__device__ __forceinline__ void split3(float a, float b, uint32_t (&p)[3])
{
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p[i]) : "f"(b), "f"(a));
        if (i < 2) a -= __uint_as_float(p[i] << 16), b -= __uint_as_float(p[i] & 0xFFFF0000u);
    }
}

// One CTA = the planes of 64 keys of one KV head (a stage of the attention kernel): K planes [key / 8][dim / 8][key % 8][8 dims], then per
// tile of 32 keys V planes [dim / 8][key / 8][dim % 8][8 keys].  Q8: int8 codes with fp16 scales per 32 dims; a value is d * q, a 19-bit
// number that its three parts hold exactly.  Keys from `len` on are zeros.
template <int HD, bool Q8>
__global__ void __launch_bounds__(256) attn_planes_kernel(const void *__restrict__ kc, const void *__restrict__ vc, const __half *__restrict__ kd,
                                                          const __half *__restrict__ vd, uint8_t *__restrict__ planes, int len, int maxSeq)
{
    using S = Shape<HD>;
    constexpr int GROUPS = CHUNK / 8, JOBS = GROUPS * (HD / 32) / 4;  // of 32 lanes x 8 values, per warp: warps 0 .. 3 K, 4 .. 7 V
    smc_grid_dep_sync();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, kvh = blockIdx.y, c = blockIdx.x;
    const bool is_v = warp >= 4;
    const float *src = static_cast<const float *>(is_v ? vc : kc) + (size_t)kvh * maxSeq * HD;
    const int8_t *codes = static_cast<const int8_t *>(is_v ? vc : kc) + (size_t)kvh * maxSeq * HD;
    const __half *ds = Q8 ? (is_v ? vd : kd) + (size_t)kvh * maxSeq * (HD / 32) : nullptr;
    uint8_t *dst = planes + ((size_t)kvh * gridDim.x + c) * S::STAGE;
#pragma unroll 2
    for (int i = 0; i < JOBS; ++i) {
        const int j = (warp & 3) * JOBS + i, kg = j % GROUPS, key0 = c * CHUNK + 8 * kg, dim0 = 32 * (j / GROUPS);
        float v[8] = {};
        if (is_v) {  // eight keys of one dim
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (key0 + u < len) {
                    if constexpr (Q8) v[u] = __half2float(ds[(size_t)(key0 + u) * (HD / 32) + dim0 / 32]) * (float)codes[(size_t)(key0 + u) * HD + dim0 + lane];
                    else v[u] = src[(size_t)(key0 + u) * HD + dim0 + lane];
                }
        } else if (key0 + (lane & 7) < len) {  // eight dims of one key
            const size_t key = key0 + (lane & 7), at = key * HD + dim0 + 8 * (lane >> 3);
            if constexpr (Q8) {
                const uint2 raw = *reinterpret_cast<const uint2 *>(codes + at);
                const float d = __half2float(ds[key * (HD / 32) + dim0 / 32]);
#pragma unroll
                for (int u = 0; u < 8; ++u) v[u] = d * (float)(int)(int8_t)(((u < 4 ? raw.x : raw.y) >> (8 * (u & 3))) & 0xFFu);
            } else {
                const float4 a = *reinterpret_cast<const float4 *>(src + at), b = *reinterpret_cast<const float4 *>(src + at + 4);
                v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
            }
        }
        const int dim = dim0 + lane;
        const uint32_t at = is_v ? S::OFF_V + (uint32_t)(kg / (KT / 8)) * S::V_TILE + (uint32_t)((dim >> 3) * (KT / 8) * 128 + (kg % (KT / 8)) * 128 + (dim & 7) * 16)
                                 : (uint32_t)(kg * (HD / 8) * 128 + (dim0 / 8 + (lane >> 3)) * 128 + (lane & 7) * 16);
        uint32_t p[4][3];
#pragma unroll
        for (int u = 0; u < 4; ++u) split3(v[2 * u], v[2 * u + 1], p[u]);
#pragma unroll
        for (int pl = 0; pl < 3; ++pl)
            *reinterpret_cast<uint4 *>(dst + at + (uint32_t)pl * (is_v ? S::V_PLANE : S::K_PLANE)) = make_uint4(p[0][pl], p[1][pl], p[2][pl], p[3][pl]);
    }
}

template <int HD>
__global__ void __launch_bounds__(THREADS, 1)
sdpa_prefill_tc_kernel(const float *__restrict__ q, const uint8_t *__restrict__ planes, float *__restrict__ out, int T, int nh, int nkv, int pos0, float scale,
                       int *status)
{
    using S = Shape<HD>;
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t sbase = smc_smem_u32(smem);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    volatile uint32_t *abort_flag = reinterpret_cast<volatile uint32_t *>(smem + S::OFF_BAR + BARS * 8 + 4);
    auto bar = [&](int i) { return sbase + S::OFF_BAR + 8u * (uint32_t)i; };
    auto wait = [&](int i, uint32_t parity) {  // by whole warps: one lane polls
        if (lane == 0) smc_tc_wait(bar(i), parity & 1u, abort_flag, status);
        __syncwarp();
    };
    auto arrive = [&](int i) {
        __syncwarp();
        if (lane == 0) smc_mbar_arrive(bar(i));
    };
    // tensor memory is taken after the predecessor has completed and before the successor may start
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; ++i) {
            smc_mbar_init(bar(FULL_K + i), 1), smc_mbar_init(bar(EMPTY_K + i), 1);
            smc_mbar_init(bar(FULL_V + i), 1), smc_mbar_init(bar(EMPTY_V + i), 1);
        }
        smc_mbar_init(bar(S_FULL), 1), smc_mbar_init(bar(S_FREE), 8), smc_mbar_init(bar(P_FULL), 4), smc_mbar_init(bar(PV_DONE), 1), smc_mbar_init(bar(PV_DONE + 1), 1), smc_mbar_init(bar(Q_FULL), 8);
        for (int i = 0; i < 8 + 16; ++i) smc_mbar_init(bar(TM_FULL + i), 1);
        *abort_flag = 0;
        smc_fence_barrier_init();
    }
    if (warp == WARP_MMA) {
        __syncwarp();
        smc_tc_alloc(sbase + S::OFF_BAR + BARS * 8, S::COLS);
    }
    smc_tc_fence_before();
    __syncthreads();
    smc_tc_fence_after();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(smem + S::OFF_BAR + BARS * 8);

    const int h = blockIdx.x, kvh = h / (nh / nkv);
    const int t0 = (int)(gridDim.y - 1 - blockIdx.y) * ROWS;  // later rows see more keys: they start first
    const int cta_len = pos0 + min(T, t0 + ROWS), chunks = (cta_len + CHUNK - 1) / CHUNK;

    if (warp < WARP_LOAD) {
        // ---------------------------------------------------------------- softmax
        const int quarter = warp & 3, mine = warp >> 2, other = mine ^ 1;  // mine: which tile of a chunk
        const int rl = 32 * quarter + lane, row = t0 + rl;
        const uint32_t lanes = tmem + ((uint32_t)(32 * quarter) << 16);
        float *tmx = reinterpret_cast<float *>(smem + S::OFF_TM);
        float2 *cpx = reinterpret_cast<float2 *>(smem + S::OFF_CP);
        {  // half of Q's dims each
            const float *src = q + ((size_t)min(row, T - 1) * nh + h) * HD;
#pragma unroll 1
            for (int c = mine * (HD / 2); c < (mine + 1) * (HD / 2); c += 32) {
                uint32_t pl[3][16];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (row < T) v = *reinterpret_cast<const float4 *>(src + c + 4 * i);
                    uint32_t a[3], b[3];
                    split3(v.x, v.y, a), split3(v.z, v.w, b);
#pragma unroll
                    for (int p = 0; p < 3; ++p) pl[p][2 * i] = a[p], pl[p][2 * i + 1] = b[p];
                }
#pragma unroll
                for (int p = 0; p < 3; ++p) st16(lanes + S::COL_Q + (uint32_t)p * S::Q_PLANE + (uint32_t)(c / 2), pl[p]);
                uint32_t zero[16] = {};
                st16(lanes + S::COL_O + (uint32_t)c, zero), st16(lanes + S::COL_O + (uint32_t)c + 16u, zero);
                wait_st();
            }
            smc_tc_fence_before();
            arrive(Q_FULL);
        }
        const int len = row < T ? pos0 + row + 1 : 0;  // keys this row sees
        const int slice = t0 + (rl & ~15), slice_len = slice < T ? pos0 + min(T, slice + 16) : 0;
        const int last = slice_len > 0 && row < T ? (slice_len - 1) / KT : -2;  // tile after which the row is stored
        float m = -INFINITY, l = 0.f;
        auto store_rows = [&](int done) {  // rows whose last tile `done` was; later tiles, masked for them, leave l as it is
            if (!__any_sync(0xffffffffu, last == done)) return;
            const float inv = l > 0.f ? 1.0f / l : 0.f;
            float *dst = out + ((size_t)min(row, T - 1) * nh + h) * HD;
#pragma unroll 1
            for (int c = 0; c < HD; c += 32) {
                uint32_t r[2][16];
                smc_tc_ld16(lanes + S::COL_O + (uint32_t)c, r[0]);
                smc_tc_ld16(lanes + S::COL_O + (uint32_t)c + 16u, r[1]);
                smc_tc_wait_ld();
                if (last == done) {
#pragma unroll
                    for (int i = 0; i < 32; i += 4)
                        *reinterpret_cast<float4 *>(dst + c + i) =
                            make_float4(__uint_as_float(r[i >> 4][i & 15]) * inv, __uint_as_float(r[i >> 4][(i & 15) + 1]) * inv,
                                        __uint_as_float(r[i >> 4][(i & 15) + 2]) * inv, __uint_as_float(r[i >> 4][(i & 15) + 3]) * inv);
                }
                __syncwarp();
            }
        };
        float s[KT];
        auto take_scores = [&](int c) {
            wait(S_FULL, (uint32_t)c);
            smc_tc_fence_after();
#pragma unroll
            for (int i0 = 0; i0 < KT; i0 += 16) {
                uint32_t a[16], b[16];
                smc_tc_ld16(lanes + S::COL_S + (uint32_t)(mine * KT + i0), a);
                smc_tc_ld16(lanes + S::COL_S + (uint32_t)(CHUNK + mine * KT + i0), b);
                smc_tc_wait_ld();
#pragma unroll
                for (int i = 0; i < 16; ++i) s[i0 + i] = (__uint_as_float(a[i]) + __uint_as_float(b[i])) * scale;
            }
            smc_tc_fence_before();
            arrive(S_FREE);
        };
        take_scores(0);
#pragma unroll 1
        for (int c = 0; c < chunks; ++c) {
            const int t = 2 * c + mine, start = t * KT;
            if (start + KT > len) {
#pragma unroll
                for (int i = 0; i < KT; ++i)
                    if (start + i >= len) s[i] = -INFINITY;
            }
            float tm = -INFINITY;
#pragma unroll
            for (int i = 0; i < KT; ++i) tm = fmaxf(tm, s[i]);
            // the tile before: its maximum is read before this one's is posted, which tells the other thread that it may post again
            if (t > 0) {
                wait(TM_FULL + 4 * other + quarter, (uint32_t)(mine ? c : c - 1));
                m = fmaxf(m, tmx[other * ROWS + rl]);
            }
            tmx[mine * ROWS + rl] = tm;
            arrive(TM_FULL + 4 * mine + quarter);
            const float nm = fmaxf(m, tm);
            // a row that sees no key of this tile (and none before) keeps m = -inf: its weights and corrections are 0
            const bool some = nm > -INFINITY;
            const float corr = some ? expf(m - nm) : 0.f;
            float ps[4] = {0.f, 0.f, 0.f, 0.f};  // keys 8 n + 2 i, + 1: the lanes of the other kernel's fragments
            uint32_t pl[3][16];
#pragma unroll
            for (int i = 0; i < KT / 2; ++i) {
                const float a = some ? expf(s[2 * i] - nm) : 0.f, b = some ? expf(s[2 * i + 1] - nm) : 0.f;
                ps[i & 3] += a + b;
                uint32_t p[3];
                split3(a, b, p);
                pl[0][i] = p[0], pl[1][i] = p[1], pl[2][i] = p[2];
            }
            const float sum = (ps[0] + ps[1]) + (ps[2] + ps[3]);
            // a slot and a barrier per chunk parity: the other thread may be a chunk behind, but no more than that (it has posted the
            // maximum that this one waited for, one chunk ago at the latest)
            cpx[(mine * 2 + (c & 1)) * ROWS + rl] = make_float2(corr, sum);
            arrive(CP_FULL + 8 * mine + 4 * (c & 1) + quarter);
            m = nm;
            if (t > 0) {
                const int oc = mine ? c : c - 1;
                wait(CP_FULL + 8 * other + 4 * (oc & 1) + quarter, (uint32_t)(oc >> 1));
                const float2 v = cpx[(other * 2 + (oc & 1)) * ROWS + rl];
                l = fmaf(l, v.x, v.y);
            }
            l = fmaf(l, corr, sum);
            if (mine && c + 1 < chunks) take_scores(c + 1);
            if (t > 0) {
                wait(PV_DONE + other, (uint32_t)((t - 1) >> 1));
                smc_tc_fence_after();
                store_rows(t - 1);
            }
#pragma unroll
            for (int p = 0; p < 3; ++p) st16(lanes + S::COL_P + (uint32_t)(p * KT / 2), pl[p]);
            if (t > 0 && __any_sync(0xffffffffu, corr != 1.0f)) {
#pragma unroll 1
                for (int c0 = 0; c0 < HD; c0 += 64) {
                    uint32_t o[4][16];
#pragma unroll
                    for (int i = 0; i < 4; ++i) smc_tc_ld16(lanes + S::COL_O + (uint32_t)(c0 + 16 * i), o[i]);
                    smc_tc_wait_ld();
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) o[i][j] = __float_as_uint(__uint_as_float(o[i][j]) * corr);
                        st16(lanes + S::COL_O + (uint32_t)(c0 + 16 * i), o[i]);
                    }
                }
            }
            wait_st();
            smc_tc_fence_before();
            arrive(P_FULL);
            if (!mine && c + 1 < chunks) take_scores(c + 1);
        }
        if (mine) {  // the tile before is done, so this barrier is in its last phase or through with it
            wait(PV_DONE + 1, (uint32_t)(chunks - 1));
            smc_tc_fence_after();
            store_rows(2 * chunks - 1);
        }
    } else if (warp == WARP_LOAD) {
        if (lane == 0) {
            const uint8_t *src = planes + (size_t)kvh * ((pos0 + T + CHUNK - 1) / CHUNK) * S::STAGE;
            for (int c = 0; c < chunks; ++c) {
                const int st = c % STAGES;
                const uint32_t parity = (uint32_t)((c / STAGES) & 1) ^ 1u, dst = sbase + (uint32_t)st * S::STAGE;  // (a fresh barrier passes the first)
                smc_tc_wait(bar(EMPTY_K + st), parity, abort_flag, status);
                smc_mbar_expect_tx(bar(FULL_K + st), S::OFF_V);
                smc_bulk_g2s(dst, src + (size_t)c * S::STAGE, S::OFF_V, bar(FULL_K + st));
                smc_tc_wait(bar(EMPTY_V + st), parity, abort_flag, status);
                smc_mbar_expect_tx(bar(FULL_V + st), S::STAGE - S::OFF_V);
                smc_bulk_g2s(dst + S::OFF_V, src + (size_t)c * S::STAGE + S::OFF_V, S::STAGE - S::OFF_V, bar(FULL_V + st));
            }
        }
    } else if (lane == 0) {
        // ---------------------------------------------------------------- MMA issue
        constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(ROWS >> 4) << 24);
        constexpr uint32_t ID_S = IDESC | ((uint32_t)(CHUNK >> 3) << 17), ID_O = IDESC | ((uint32_t)(HD >> 3) << 17);
        constexpr int A_PART[6] = {1, 0, 2, 0, 1, 0}, B_PART[6] = {1, 2, 0, 1, 0, 0};  // smallest products first
        bool k_there = false, v_there = false;  // the next chunk's planes, as far as is known
        auto scores = [&](int c) {
            const int st = c % STAGES;
            if (!k_there) smc_tc_wait(bar(FULL_K + st), (uint32_t)(c / STAGES) & 1u, abort_flag, status);
            smc_tc_wait(bar(S_FREE), (uint32_t)(c & 1) ^ 1u, abort_flag, status);
            smc_tc_fence_after();
            k_there = smc_mbar_test(bar(FULL_K + (c + 1) % STAGES), (uint32_t)((c + 1) / STAGES) & 1u);
            const uint64_t k0 = desc(sbase + (uint32_t)st * S::STAGE, 128, HD / 8 * 128);
#pragma unroll
            for (int ks = 0; ks < HD / 16; ++ks) {
                const uint32_t d = tmem + S::COL_S + (uint32_t)((ks & 1) * CHUNK);
#pragma unroll
                for (int i = 0; i < 6; ++i)
                    mma_ta(d, tmem + S::COL_Q + (uint32_t)A_PART[i] * S::Q_PLANE + (uint32_t)ks * 8u,
                           k0 + (uint64_t)((uint32_t)B_PART[i] * S::K_PLANE + (uint32_t)ks * 256u) / 16u, ID_S, ks > 1 || i > 0 ? 1u : 0u);
            }
            smc_tc_commit(bar(S_FULL));
            smc_tc_commit(bar(EMPTY_K + st));
        };
        smc_tc_wait(bar(Q_FULL), 0u, abort_flag, status);
        smc_tc_fence_after();
        scores(0);
#pragma unroll 1
        for (int c = 0; c < chunks; ++c) {
            const int st = c % STAGES;
            v_there = smc_mbar_test(bar(FULL_V + st), (uint32_t)(c / STAGES) & 1u);
            if (c + 1 < chunks) scores(c + 1);
            if (!v_there) smc_tc_wait(bar(FULL_V + st), (uint32_t)(c / STAGES) & 1u, abort_flag, status);
#pragma unroll 1
            for (int u = 0; u < 2; ++u) {
                smc_tc_wait(bar(P_FULL), (uint32_t)u, abort_flag, status);
                smc_tc_fence_after();
                const uint64_t v0 = desc(sbase + (uint32_t)st * S::STAGE + S::OFF_V + (uint32_t)u * S::V_TILE, 128, KT / 8 * 128);
#pragma unroll
                for (int j = 0; j < KT / 16; ++j)
#pragma unroll
                    for (int i = 0; i < 6; ++i)
                        mma_ta(tmem + S::COL_O, tmem + S::COL_P + (uint32_t)(A_PART[i] * KT / 2 + j * 8),
                               v0 + (uint64_t)((uint32_t)B_PART[i] * S::V_PLANE + (uint32_t)j * 256u) / 16u, ID_O, 1u);
                smc_tc_commit(bar(PV_DONE + u));
            }
            smc_tc_commit(bar(EMPTY_V + st));
        }
    }
    smc_tc_fence_before();
    __syncthreads();
    if (warp == WARP_MMA) {
        __syncwarp();
        smc_tc_dealloc(tmem, S::COLS);
    }
}

}  // namespace

static size_t stage_bytes(int hd) { return hd == 128 ? Shape<128>::STAGE : Shape<64>::STAGE; }

// One buffer for all lengths that the cache can have, up to a limit: nothing grows with the context and nothing is freed before the object.
// Without one (a full device) the calls take the mma.sync kernel.  cudaMalloc touches no stream, so the thread may ask for it while it, or
// another, captures one.
void smc_attn_planes_reserve(smc_attn_planes *planes, int kvHeads, int headDim, int maxSeq)
{
    if (planes->reserved) return;
    planes->reserved = true;
    const size_t want = (size_t)kvHeads * ((maxSeq + (size_t)CHUNK - 1) / CHUNK) * stage_bytes(headDim);
    planes->bytes = want < ATTN_PLANES_MOST ? want : ATTN_PLANES_MOST;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (cudaMalloc(&planes->d, planes->bytes) != cudaSuccess) {
        cudaGetLastError();
        planes->d = nullptr, planes->bytes = 0;
    }
    cudaThreadExchangeStreamCaptureMode(&mode);
}

int smc_launch_sdpa_prefill_tc(smc_ctx *ctx, smc_attn_planes *own, const float *q, const void *kc, const void *vc, const __half *kd, const __half *vd, float *out,
                               int T, int nh, int nkv, int hd, int pos0, int maxSeq, float scale, cudaStream_t s)
{
    const int chunks = (pos0 + T + CHUNK - 1) / CHUNK;
    std::lock_guard<std::mutex> lock(ctx->mu_attn);  // two threads on the object's stream: not one's attention between the other's two launches
    smc_attn_planes_reserve(own, nkv, hd, maxSeq);
    if ((size_t)nkv * chunks * stage_bytes(hd) > own->bytes) return SMC_E_UNSUPPORTED;
    uint8_t *planes = own->d;
    auto go = [&](auto split, auto kernel, size_t smem) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        smc_launch_dep(ctx->use_pdl, split, dim3(chunks, nkv), dim3(256), 0, s, kc, vc, kd, vd, planes, pos0 + T, maxSeq);
        smc_launch_dep(ctx->use_pdl, kernel, dim3(nh, (T + ROWS - 1) / ROWS), dim3(THREADS), smem, s, q, planes, out, T, nh, nkv, pos0, scale, ctx->d_status);
    };
    if (hd == 128) kd ? go(attn_planes_kernel<128, true>, sdpa_prefill_tc_kernel<128>, Shape<128>::SMEM) : go(attn_planes_kernel<128, false>, sdpa_prefill_tc_kernel<128>, Shape<128>::SMEM);
    else kd ? go(attn_planes_kernel<64, true>, sdpa_prefill_tc_kernel<64>, Shape<64>::SMEM) : go(attn_planes_kernel<64, false>, sdpa_prefill_tc_kernel<64>, Shape<64>::SMEM);
    SMC_LAUNCH_CHECK(ctx);
    return SMC_OK;
}
