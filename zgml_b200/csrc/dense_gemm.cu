// Dense prefill matmul for the sequence-model LINEAR op on the 5th-generation tensor cores:
//   dst[M, N] = bf16(src)[M, K] * W[N, K]^T (+ bias), W stored bfloat16 row-major (the checkpoint's [out, in]).
//
//   * tcgen05.mma.cta_group::1.kind::f16 on BF16 operands, one 128 x 128 fp32 accumulator per CTA in TMEM, issued by the
//     elected lane of a warp; K advances 64 (one 128-byte swizzle row) per pipeline stage.
//   * BOTH operands arrive by TMA (cp.async.bulk.tensor.2d, 128B swizzle) straight into the canonical K-major layout: the
//     weight matrix as it lies in the arena (out-of-range rows / k are zero-filled by the copy engine), the activations
//     from a bf16 scratch that a small conversion kernel fills (one rounding per activation; accumulation stays fp32).
//   * 6-stage mbarrier ring (32 KB per stage): TMA warp -> MMA warp -> (tcgen05.commit) -> stage free.  Four epilogue warps
//     read the accumulator (tcgen05.ld 32x32b), transpose 32 x 32 blocks through the idle stage memory, add the bias and
//     write 128-byte row segments.
//   * Every wait is bounded: a barrier that does not flip within ~1 s of polling is counted
//     (zg_dense_gemm_timeouts) and the CTA drains — its roles all give up the same way — frees its TMEM and returns.
//
// Used when the session keeps bfloat16 weights and M > 8 (decode rows stream the weights through the row kernels of
// seqops.cu); float32 sessions' products of many rows are split_gemm.cu's.
#include "split_tc.cuh"

#include <algorithm>

namespace {

constexpr uint32_t BM = 128, BN = 128, BK = 64;
constexpr uint32_t kTileA = BM * BK * 2, kTileB = BN * BK * 2, kStage = kTileA + kTileB;
constexpr uint32_t kStages = 6;
constexpr uint32_t kThreads = 192;   // warp 0: TMA, warp 1: MMA + TMEM, warps 2-5: epilogue
constexpr uint32_t kTmemCols = 128;
constexpr uint32_t kSmem = kStages * kStage + 1024 + 256;

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t c0, uint32_t c1, uint32_t c2, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar) : "memory");
}
// K-major, 128-byte swizzle, 8-row groups 1024 B apart
__device__ __forceinline__ uint64_t make_desc(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// D[tmem] (+)= A[shared] B[shared], bf16
__device__ __forceinline__ void mma_bf16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
// f32 rows -> dense bf16 [Mp][Kp] (zero padding), two k per thread
// (ctl: the rows are those of a per-sequence state buffer, `slot_stride` elements per slot; the slot is the control word's)
// (rows_from > 0: rows from position + rows_from on are not wanted, up to the end of their 128-row tile)
// blockIdx.z: a batch of sources x_hs apart, each with its own padded rows in `out`
__global__ void k_to_bf16(const float* __restrict__ x, uint32_t x_rs, uint32_t* __restrict__ out, uint32_t kp2, uint32_t M, uint32_t K, const float* __restrict__ ctl,
                          uint32_t slot_stride, uint32_t rows_from, uint32_t x_hs) {
    const uint32_t m = blockIdx.y;
    if (rows_from && m / BM * BM >= (uint32_t)reinterpret_cast<const int*>(ctl)[ZG_CTL_POS] + rows_from) return;
    if (ctl) x += (size_t)reinterpret_cast<const int*>(ctl)[ZG_CTL_SLOT] * slot_stride;
    x += (size_t)blockIdx.z * x_hs;
    out += (size_t)blockIdx.z * gridDim.y * kp2;
    for (uint32_t k2 = blockIdx.x * blockDim.x + threadIdx.x; k2 < kp2; k2 += gridDim.x * blockDim.x) {
        const uint32_t k = 2 * k2;
        const float a = (m < M && k < K) ? x[(size_t)m * x_rs + k] : 0.0f;
        const float b = (m < M && k + 1 < K) ? x[(size_t)m * x_rs + k + 1] : 0.0f;
        uint32_t r;
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
        out[(size_t)m * kp2 + k2] = r;
    }
}

// the epilogue's activation (the kinds of the ACTIVATION op, shifted by one: 0 is none), a compile-time kind: 128 outputs per
// epilogue thread pass it one after the other, so what counts is straight-line code whose chains interleave.  (A switch inside the
// loop cost 340 cycles per output.)  Exponentials and quotients are the fast intrinsics: the product's inputs are bfloat16.
// The exact GELU takes erf from Abramowitz and Stegun, Handbook of Mathematical Functions, formula 7.1.26 (absolute error below
// 1.5e-7): 1 - erf(x) = (a1 t + ... + a5 t^5) exp(-x^2), t = 1 / (1 + p x), x >= 0.
template <int ACT>
__device__ __forceinline__ float gemm_act(float z, float p) {
    if (ACT == 1) { const float r = fmaxf(z, 0.0f); return r * r; }
    if (ACT == 2) return __fdividef(z, 1.0f + __expf(-z));
    if (ACT == 3) return 0.5f * z * (1.0f + tanhf(0.7978845608028654f * fmaf(0.044715f * z * z, z, z)));
    if (ACT == 4) return fmaxf(z, 0.0f);
    if (ACT == 5) return p * tanhf(z / p);
    if (ACT == 6) {
        const float x = fabsf(z) * 0.7071067811865476f, t = __fdividef(1.0f, fmaf(0.3275911f, x, 1.0f));
        const float poly = t * fmaf(t, fmaf(t, fmaf(t, fmaf(t, 1.061405429f, -1.453152027f), 1.421413741f), -0.284496736f), 0.254829592f);
        const float tail = poly * __expf(-x * x);      // 1 - erf(x)
        return 0.5f * z * (z < 0.0f ? tail : 2.0f - tail);
    }
    return z;
}
struct GemmParams {
    float* out;
    const __nv_bfloat16* bias;
    uint32_t M, N, K, out_rs, out_vec4;
    uint32_t act;            // applied after the bias: 0 none, 1 relu^2, 2 silu, 3 gelu (tanh form), 4 relu, 5 smooth cap act_p * tanh(z / act_p), 6 gelu (erf form)
    float act_p;
    uint32_t act_lo, act_hi; // the columns it applies to
    const int* ctl;          // kPlain with rows_from: tiles from row position + rows_from on are skipped
    uint32_t rows_from;
    uint32_t heads, n_last, a_rows, out_hs;   // kBatched: heads, rows of the last head's matrix, padded source rows per head, columns between the heads' outputs
};

// kBatched: blockIdx.z names a head with source rows, weight rows and output columns of its own (all in one tensor each).  A tile at the
// end of a head reads on into the next head's weight rows; those columns are not written.
// PAIRS: weight rows 2n and 2n + 1 are a gate and what it multiplies: out[., n] = act(gate) * up.
enum { kPlain = 0, kBatched = 1 };
template <int MODE, int ACT, bool PAIRS>        // ACT: the activation of the epilogue (GemmParams::act; one instantiation each)
__global__ void __launch_bounds__(kThreads, 1)
dense_gemm_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const GemmParams p) {
    const uint32_t head = MODE == kBatched ? blockIdx.z : 0, N = MODE == kBatched && head + 1 == p.heads ? p.n_last : p.N;
    if (MODE == kBatched && blockIdx.x * BN >= N) return;
    if (MODE == kPlain && p.rows_from && blockIdx.y * BM >= (uint32_t)p.ctl[ZG_CTL_POS] + p.rows_from) return;
    float* const outp = p.out + (MODE == kBatched ? (size_t)head * p.out_hs : 0);
    extern __shared__ uint8_t dsm_raw[];
    const uint32_t base = (smem_u32(dsm_raw) + 1023u) & ~1023u;
    const uint32_t bars = base + kStages * kStage;
    const uint32_t full = bars, empty = bars + 8 * kStages, tmem_full = bars + 16 * kStages, tmem_slot = tmem_full + 8;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t tile_n = blockIdx.x, tile_m = blockIdx.y;
    const uint32_t n_k = (p.K + BK - 1) / BK;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < kStages; s++) { mbar_init(full + 8 * s, 1); mbar_init(empty + 8 * s, 1); }
        mbar_init(tmem_full, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "n"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    uint32_t tmem_base;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot));

    if (warp == 0) {
        if (lane == 0) {
            uint32_t fills = 0;
            for (uint32_t kt = 0; kt < n_k; kt++) {
                const uint32_t s = kt % kStages, ph = (kt / kStages) & 1;
                if (!mbar_wait(empty + 8 * s, ph ^ 1)) break;
                mbar_expect_tx(full + 8 * s, kStage);
                tma_2d(base + s * kStage, &tmap_a, kt * BK, head * p.a_rows + tile_m * BM, full + 8 * s);
                tma_2d(base + s * kStage + kTileA, &tmap_b, kt * BK, head * p.N + tile_n * BN, full + 8 * s);
                fills++;
            }
            // the copies that are under way land before the CTA's shared memory goes, whatever gave up
            for (uint32_t i = 0; i < min(fills, (uint32_t)kStages); i++) mbar_wait(full + 8 * i, ((fills - 1 - i) / kStages) & 1);
        }
    } else if (warp == 1) {
        // instruction descriptor (kind::f16): D = F32, A = B = BF16, both K-major, N = BN, M = 128
        constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((BN >> 3) << 17) | ((128u >> 4) << 24);
        const bool leader = elect_one();
        uint32_t issued = 0;
        for (uint32_t kt = 0; kt < n_k; kt++) {
            const uint32_t s = kt % kStages, ph = (kt / kStages) & 1;
            if (!__all_sync(0xffffffffu, mbar_wait(full + 8 * s, ph))) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (uint32_t k = 0; k < BK / 16; k++)
                if (leader) mma_bf16(tmem_base, make_desc(base + s * kStage + k * 32), make_desc(base + s * kStage + kTileA + k * 32), idesc, (kt | k) ? 1u : 0u);
            if (leader) mma_commit(empty + 8 * s);
            if (leader && kt + 1 == n_k) mma_commit(tmem_full);
            issued = kt + 1;
        }
        // products under way end before their accumulator goes
        if (issued < n_k && issued) mbar_wait(empty + 8 * ((issued - 1) % kStages), ((issued - 1) / kStages) & 1);
        __syncwarp();
    } else {
        // ── epilogue: warp w may touch TMEM lanes 32 (w % 4) .. + 31 ──
        const uint32_t ew = warp - 2, quarter = warp & 3;
        const bool ok = mbar_wait(tmem_full, 0);       // (what the other roles gave up on does not arrive here either)
        if (!ok && lane == 0) count_timeout();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t m_base = tile_m * BM + quarter * 32;
        if (!ok) {      // outputs that are not numbers, instead of what was there before
            const uint32_t per = PAIRS ? 2 : 1, n1 = min(N, (tile_n + 1) * BN) / per;
            for (uint32_t n = tile_n * BN / per + lane; n < n1; n += 32)
                for (uint32_t m = m_base; m < min(p.M, m_base + 32); m++) outp[(size_t)m * p.out_rs + n] = __int_as_float(0x7fc00000);
        }
        uint4* tb = reinterpret_cast<uint4*>(dsm_raw + (base - smem_u32(dsm_raw)) + ew * (32 * 36 * 4));   // the stages are idle now
#pragma unroll 1
        for (uint32_t c0 = 0; ok && c0 < BN; c0 += 32) {
            uint32_t v[32];
            const uint32_t taddr = tmem_base + ((quarter * 32) << 16) + c0;
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                  "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
                  "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
                  "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                : "r"(taddr));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int i = 0; i < 8; i++) tb[lane * 9 + i] = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            __syncwarp();
            const uint32_t n0 = tile_n * BN + c0;
            const bool acts = ACT && (MODE != kBatched || head + 1 == p.heads), some = acts && n0 < p.act_hi && n0 + 32 > p.act_lo;     // uniform: whether any of these columns takes the activation
            auto finish = [&](float z, uint32_t n) {
                if (!ACT) return z;
                const float a = gemm_act<ACT>(z, p.act_p);
                return acts && n >= p.act_lo && n < p.act_hi ? a : z;
            };
            if (PAIRS) {
                if (p.out_vec4 && n0 + 32 <= N) {
                    const uint32_t nn = n0 + 4 * (lane & 7);
#pragma unroll
                    for (int it = 0; it < 8; it++) {
                        const uint32_t rr = it * 4 + (lane >> 3), mm = m_base + rr;
                        const uint4 o = tb[rr * 9 + (lane & 7)];
                        const float2 f = make_float2(gemm_act<ACT>(__uint_as_float(o.x), p.act_p) * __uint_as_float(o.y), gemm_act<ACT>(__uint_as_float(o.z), p.act_p) * __uint_as_float(o.w));
                        if (mm < p.M) *reinterpret_cast<float2*>(outp + (size_t)mm * p.out_rs + nn / 2) = f;
                    }
                } else if (lane < 16 && n0 + 2 * lane + 1 < N) {
                    const uint32_t* tw = reinterpret_cast<const uint32_t*>(tb);
                    for (int rr = 0; rr < 32; rr++)
                        if (m_base + rr < p.M)
                            outp[(size_t)(m_base + rr) * p.out_rs + n0 / 2 + lane] = gemm_act<ACT>(__uint_as_float(tw[rr * 36 + 2 * lane]), p.act_p) * __uint_as_float(tw[rr * 36 + 2 * lane + 1]);
                }
            } else if (n0 < N) {
                if (p.out_vec4 && n0 + 32 <= N) {
                    const uint32_t nn = n0 + 4 * (lane & 7);
                    float b[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                    if (p.bias) for (int j = 0; j < 4; j++) b[j] = __bfloat162float(p.bias[nn + j]);
                    if (!ACT || some) {
#pragma unroll
                    for (int it = 0; it < 8; it++) {
                        const uint32_t rr = it * 4 + (lane >> 3), mm = m_base + rr;
                        const uint4 o = tb[rr * 9 + (lane & 7)];
                        const float4 f = make_float4(finish(__uint_as_float(o.x) + b[0], nn), finish(__uint_as_float(o.y) + b[1], nn + 1), finish(__uint_as_float(o.z) + b[2], nn + 2),
                                                     finish(__uint_as_float(o.w) + b[3], nn + 3));
                        if (mm < p.M) *reinterpret_cast<float4*>(outp + (size_t)mm * p.out_rs + nn) = f;
                    }
                    } else {
#pragma unroll
                    for (int it = 0; it < 8; it++) {
                        const uint32_t rr = it * 4 + (lane >> 3), mm = m_base + rr;
                        const uint4 o = tb[rr * 9 + (lane & 7)];
                        const float4 f = make_float4(__uint_as_float(o.x) + b[0], __uint_as_float(o.y) + b[1], __uint_as_float(o.z) + b[2], __uint_as_float(o.w) + b[3]);
                        if (mm < p.M) *reinterpret_cast<float4*>(outp + (size_t)mm * p.out_rs + nn) = f;
                    }
                    }
                } else if (n0 + lane < N) {
                    const uint32_t* tw = reinterpret_cast<const uint32_t*>(tb);
                    const float b = p.bias ? __bfloat162float(p.bias[n0 + lane]) : 0.0f;
                    for (int rr = 0; rr < 32; rr++)
                        if (m_base + rr < p.M) outp[(size_t)(m_base + rr) * p.out_rs + n0 + lane] = finish(__uint_as_float(tw[rr * 36 + lane]) + b, n0 + lane);
                }
            }
            __syncwarp();
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(kTmemCols) : "memory");
}

// Expert products of MOE_FFN: out[row, n] = sum_k x[row, k] W_e[n, k] for rows sorted by expert, one run of at most 256 rows of one expert per blockIdx.y.
//
// The weights are the 128-row operand and the run's rows the N operand, of as many columns as the run has rows (rounded up to 16): every weight is read
// once per run, and what is computed for padding is less than 16 rows (whole 128-row tiles of tokens were a third padding at 16 experts of 128 rows each,
// and read the weights again for it).  DUAL: two weight matrices against the same rows, gate and up, and out = bf16(act(gate) up), so that neither
// product goes through memory.
// Where there are more tiles than SMs, a CTA per SM walks them: the next tile's operands are on their way while this one's products end, and its products run while this one
// is written out, where two accumulators have room.  1024 tokens, two of 16 experts, 2048 x 2048: the op 125 us with a CTA per tile, 120 walked, 117 with the down product by
// 256 rows; two of 8 experts, 1024 x 1024 61.6 -> 53.8; 700 tokens, one of 16, 1600 / 296 43.0 -> 39.8.  What bounds it is what the SMs take in: 403 MB of weights from memory and
// 240 MB of runs' rows from the L2 (64 tokens, the same weights: 87 us, of which the two products take some 65 at 6.2 TB/s).
constexpr uint32_t kExpertThreads = 320;          // warp 0: TMA, warp 1: MMA + TMEM, warps 2-9: epilogue
constexpr uint32_t kExpertRows = 32;              // rows of x per copy
constexpr uint32_t kExpertRing = 216 * 1024, kExpertSmem = kExpertRing + 1024 + 256, kExpertStages = 8;
struct ExpertParams {
    void* out; const ZgExpertSegment* segments;
    uint32_t N, K, runs;                           // runs: room in `segments`; those with rows come first
    float limit, alpha, up_offset;
};
enum { kExpertDual, kExpertWide, kExpertOne };      // gate and up; 256 and 128 rows of one matrix
// LOOP: a CTA per SM takes every gridDim.x-th tile of all runs; otherwise a CTA is (tile, run), and done after it
template <int MODE, bool LOOP>
__global__ void __launch_bounds__(kExpertThreads, 1)
k_expert_gemm(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_w2, const ExpertParams p) {
    constexpr bool DUAL = MODE == kExpertDual, PAIR = MODE != kExpertOne;      // PAIR: two 128-row operands
    constexpr uint32_t ROWS = MODE == kExpertWide ? 2 * BM : BM;               // of the output's columns that a tile covers
    pdl_enter();
    const uint32_t n_k = (p.K + BK - 1) / BK, n_f = (p.N + ROWS - 1) / ROWS;
    const ZgExpertSegment first = p.segments[LOOP ? min(blockIdx.x / n_f, p.runs - 1) : blockIdx.y];      // of the first tile: on its way with the others
    if (!LOOP && first.rows <= 0) return;          // uniform over the CTA, before any barrier or TMEM allocation
    auto run_of = [&](uint32_t t) { return !LOOP || t == blockIdx.x ? first : p.segments[t / n_f]; };
    extern __shared__ uint8_t dsm_raw[];
    __shared__ uint32_t live, longest;             // runs with rows, rows of the longest
    const uint32_t base = (smem_u32(dsm_raw) + 1023u) & ~1023u, bars = base + kExpertRing;
    const uint32_t full = bars, empty = bars + 8 * kExpertStages, tmem_full = bars + 16 * kExpertStages, tmem_empty = tmem_full + 16, tmem_slot = tmem_empty + 16;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < kExpertStages; s++) { mbar_init(full + 8 * s, 1); mbar_init(empty + 8 * s, 1); }
        for (uint32_t i = 0; i < 2; i++) { mbar_init(tmem_full + 8 * i, 1); mbar_init(tmem_empty + 8 * i, 8); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(tmem_slot) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (LOOP && warp == 2) {
        uint32_t n = 0, mx = 0;
        for (uint32_t i = lane; i < p.runs; i += 32) {
            const uint32_t rows = (uint32_t)max(p.segments[i].rows, 0);
            n += rows > 0;
            mx = max(mx, rows);
        }
        n = __reduce_add_sync(0xffffffffu, n);
        mx = __reduce_max_sync(0xffffffffu, mx);
        if (lane == 0) { live = n; longest = mx; }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    uint32_t tmem;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(tmem_slot));
    constexpr uint32_t kWeights = (PAIR ? 2 : 1) * kTileA;
    const uint32_t tiles = LOOP ? live * n_f : n_f, most = LOOP ? longest : (uint32_t)first.rows;
    const uint32_t stage_bytes = kWeights + (most + kExpertRows - 1) / kExpertRows * (kExpertRows * BK * 2), stages = min(kExpertStages, kExpertRing / stage_bytes);
    // accumulators: two where both fit the 512 columns, so that a tile's products run while the one before is written out
    const bool two = (PAIR ? 4 : 2) * ((most + 15) / 16 * 16) <= 512;
    const uint32_t up_at = two && PAIR ? 128 : 256;              // the second matrix's columns; the other accumulator lies 256 columns on

    if (warp == 0) {
        if (lane == 0) {
            uint32_t s = 0, ph = 1, fills = 0;
            bool ok = true;
            for (uint32_t t = blockIdx.x; ok && t < tiles; t += gridDim.x) {
                const ZgExpertSegment seg = run_of(t);
                const uint32_t f0 = t % n_f * ROWS, copies = ((uint32_t)seg.rows + kExpertRows - 1) / kExpertRows;
                for (uint32_t kt = 0; kt < n_k; kt++) {
                    ok = mbar_wait(empty + 8 * s, ph);
                    if (!ok) break;
                    const uint32_t at = base + s * stage_bytes;
                    mbar_expect_tx(full + 8 * s, kWeights + copies * (kExpertRows * BK * 2));
                    tma_load_3d(at, &tmap_w, kt * BK, f0, (uint32_t)seg.expert, full + 8 * s);
                    if (PAIR) tma_load_3d(at + kTileA, &tmap_w2, kt * BK, DUAL ? f0 : f0 + BM, (uint32_t)seg.expert, full + 8 * s);
                    for (uint32_t c = 0; c < copies; c++) tma_2d(at + kWeights + c * (kExpertRows * BK * 2), &tmap_x, kt * BK, (uint32_t)seg.start + c * kExpertRows, full + 8 * s);
                    fills++;
                    if (++s == stages) { s = 0; ph ^= 1; }
                }
            }
            // the copies that are under way land before the CTA's shared memory goes, whatever gave up
            for (uint32_t i = 0; i < min(fills, stages); i++) mbar_wait(full + 8 * i, ((fills - 1 - i) / stages) & 1);
        }
    } else if (warp == 1) {
        const bool leader = elect_one();
        uint32_t s = 0, ph = 0, i = 0, last = 0, last_ph = 0;
        bool ok = true;
        for (uint32_t t = blockIdx.x; ok && t < tiles; t += gridDim.x, i++) {
            // instruction descriptor (kind::f16): D = F32, A = B = BF16, both K-major, N = the run's rows, M = 128
            const uint32_t n = (uint32_t)run_of(t).rows, idesc = (1u << 4) | (1u << 7) | (1u << 10) | (((n + 15) / 16 * 2) << 17) | ((128u >> 4) << 24);
            const uint32_t acc = two ? i & 1 : 0, use = two ? i >> 1 : i, d = tmem + acc * 256;
            if (use) ok = __all_sync(0xffffffffu, mbar_wait(tmem_empty + 8 * acc, (use - 1) & 1));
            for (uint32_t kt = 0; ok && kt < n_k; kt++) {
                ok = __all_sync(0xffffffffu, mbar_wait(full + 8 * s, ph));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t at = base + s * stage_bytes;
#pragma unroll
                for (uint32_t k = 0; k < BK / 16; k++)
                    if (leader) {
                        const uint64_t x = make_desc(at + kWeights + k * 32);
                        mma_bf16(d, make_desc(at + k * 32), x, idesc, (kt | k) ? 1u : 0u);
                        if (PAIR) mma_bf16(d + up_at, make_desc(at + kTileA + k * 32), x, idesc, (kt | k) ? 1u : 0u);
                    }
                if (leader) mma_commit(empty + 8 * s);
                if (leader && kt + 1 == n_k) mma_commit(tmem_full + 8 * acc);
                last = empty + 8 * s; last_ph = ph;
                if (++s == stages) { s = 0; ph ^= 1; }
            }
        }
        if (!ok && last) mbar_wait(last, last_ph);      // products under way end before their accumulators go
        __syncwarp();
    } else {
        // TMEM lane = output column of the tile's 128, TMEM column = row of the run; the two warps of a quarter take 16 rows each in turn
        const uint32_t quarter = warp & 3, half = (warp - 2) >> 2;
        uint32_t i = 0;
        bool ok = true;
        for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x, i++) {
            const ZgExpertSegment seg = run_of(t);
            const uint32_t n = (uint32_t)seg.rows, f = t % n_f * ROWS + quarter * 32 + lane, acc = two ? i & 1 : 0, use = two ? i >> 1 : i;
            if (ok) {
                ok = __all_sync(0xffffffffu, mbar_wait(tmem_full + 8 * acc, use & 1));       // (what the other roles gave up on does not arrive here either)
                if (!ok && lane == 0) count_timeout();
            }
            if (!ok) {      // the outputs of this tile and of those after it are not numbers
                for (uint32_t c = half; f < p.N && c < n; c += 2) {
                    const size_t at = ((size_t)seg.start + c) * p.N + f;
                    if (DUAL) reinterpret_cast<__nv_bfloat16*>(p.out)[at] = __float2bfloat16_rn(__int_as_float(0x7fc00000));
                    else {
                        reinterpret_cast<float*>(p.out)[at] = __int_as_float(0x7fc00000);
                        if (PAIR && f + BM < p.N) reinterpret_cast<float*>(p.out)[at + BM] = __int_as_float(0x7fc00000);
                    }
                }
                continue;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (uint32_t c0 = 16 * half; c0 < n; c0 += 32) {
                uint32_t g[16], u[16];
                const uint32_t addr = tmem + acc * 256 + ((quarter * 32) << 16) + c0;
                tmem_ld(addr, g);
                if (PAIR) tmem_ld(addr + up_at, u);
                tmem_wait_ld(g);
                if (PAIR) tmem_wait_ld(u);
#pragma unroll
                for (uint32_t j = 0; j < 16; j++) {
                    if (c0 + j >= n || f >= p.N) continue;
                    const size_t at = ((size_t)seg.start + c0 + j) * p.N + f;
                    if (DUAL) {
                        const float gv = fminf(__uint_as_float(g[j]), p.limit), uv = fminf(fmaxf(__uint_as_float(u[j]), -p.limit), p.limit);
                        reinterpret_cast<__nv_bfloat16*>(p.out)[at] = __float2bfloat16_rn(gv * sigmoidf_(p.alpha * gv) * (uv + p.up_offset));
                    } else {
                        reinterpret_cast<float*>(p.out)[at] = __uint_as_float(g[j]);
                        if (PAIR && f + BM < p.N) reinterpret_cast<float*>(p.out)[at + BM] = __uint_as_float(u[j]);
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(tmem_empty + 8 * acc) : "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

EncodeTiledFn g_encode = nullptr;
bool g_attr_set = false;
constexpr int kActs = 7;
typedef void (*GemmKernel)(const CUtensorMap, const CUtensorMap, const GemmParams);
#define ZG_ACTS(MODE_, PAIRS_)                                                                                                                           \
    {dense_gemm_kernel<MODE_, 0, PAIRS_>, dense_gemm_kernel<MODE_, 1, PAIRS_>, dense_gemm_kernel<MODE_, 2, PAIRS_>, dense_gemm_kernel<MODE_, 3, PAIRS_>, \
     dense_gemm_kernel<MODE_, 4, PAIRS_>, dense_gemm_kernel<MODE_, 5, PAIRS_>, dense_gemm_kernel<MODE_, 6, PAIRS_>}
const GemmKernel g_kernel[2][kActs] = {ZG_ACTS(kPlain, false), ZG_ACTS(kPlain, true)};   // [pairs][activation]
#undef ZG_ACTS
typedef void (*ExpertKernel)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const ExpertParams);
const ExpertKernel g_expert[3][2] = {{k_expert_gemm<kExpertDual, false>, k_expert_gemm<kExpertDual, true>}, {k_expert_gemm<kExpertWide, false>, k_expert_gemm<kExpertWide, true>},
                                     {k_expert_gemm<kExpertOne, false>, k_expert_gemm<kExpertOne, true>}};      // [mode][loop]
GemmKernel batched_kernel(uint32_t act) {      // the activations a batched product's last head can have
    return act == 0 ? dense_gemm_kernel<kBatched, 0, false> : act == 5 ? dense_gemm_kernel<kBatched, 5, false> : (GemmKernel)nullptr;
}

bool prepare() {
    if (!g_encode) {
        g_encode = encode_tiled();
        if (!g_encode) { zg_set_error("cuTensorMapEncodeTiled entry point not available"); return false; }
    }
    if (!g_attr_set) {
        cudaError_t e = cudaSuccess;
        for (int k = 0; k < 6 && e == cudaSuccess; k++) e = cudaFuncSetAttribute(g_expert[k / 2][k % 2], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kExpertSmem);
        for (int k = 0; k < 2 * kActs && e == cudaSuccess; k++) e = cudaFuncSetAttribute(g_kernel[k / kActs][k % kActs], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
        for (uint32_t k = 0; k < 6 && e == cudaSuccess; k += 5) e = cudaFuncSetAttribute(batched_kernel(k), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
        if (e != cudaSuccess) { zg_set_error("cudaFuncSetAttribute(dense_gemm) failed: %s", cudaGetErrorString(e)); return false; }
        g_attr_set = true;
    }
    return true;
}

}  // namespace

// The tensor path takes whole-tile-sized problems whose weight rows TMA can address (16-byte aligned base and pitch).
bool zg_dense_gemm_usable(const void* w_bf16, uint32_t M, uint32_t N, uint32_t K) {
    return M > 8 && N >= 8 && K >= 64 && K % 8 == 0 && (reinterpret_cast<uintptr_t>(w_bf16) & 15) == 0;
}
// bf16 copy of the activations: [round_up(M, 128)][round_up(K, 64)], counted in f32 slots
size_t zg_dense_gemm_scratch_elems(uint32_t M, uint32_t K) {
    return (size_t)((M + BM - 1) / BM * BM) * ((K + BK - 1) / BK * BK) / 2;
}
unsigned int zg_dense_gemm_timeouts() { return tc_timeouts(); }

bool zg_dense_gemm_launch(const void* w_bf16, const void* bias_bf16, const float* src, float* dst, uint32_t M, uint32_t N, uint32_t K,
                          uint32_t src_rs, uint32_t dst_rs, float* scratch, cudaStream_t st, uint32_t act, float act_p, uint32_t act_lo, uint32_t act_hi, const float* ctl, uint32_t slot_stride, bool pairs,
                          uint32_t rows_from) {
    if (!prepare()) return false;
    if (pairs) N *= 2;                                   // weight rows
    const uint32_t Kp = (K + BK - 1) / BK * BK, Mp = (M + BM - 1) / BM * BM;
    uint32_t* xb = reinterpret_cast<uint32_t*>(scratch);
    k_to_bf16<<<dim3((Kp / 2 + 255) / 256, Mp), 256, 0, st>>>(src, src_rs, xb, Kp / 2, M, K, ctl, slot_stride, rows_from, 0u);
    ZG_COUNT_LAUNCH();
    CUtensorMap map_a, map_b;
    const cuuint32_t estr[2] = {1, 1};
    {
        const cuuint64_t gdim[2] = {Kp, Mp};
        const cuuint64_t gstride[1] = {(cuuint64_t)Kp * 2};
        const cuuint32_t box[2] = {BK, BM};
        CUresult r = g_encode(&map_a, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, xb, gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) { zg_set_error("cuTensorMapEncodeTiled(activations) failed (%d)", (int)r); return false; }
    }
    {
        const cuuint64_t gdim[2] = {K, N};
        const cuuint64_t gstride[1] = {(cuuint64_t)K * 2};
        const cuuint32_t box[2] = {BK, BN};
        CUresult r = g_encode(&map_b, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(w_bf16), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) { zg_set_error("cuTensorMapEncodeTiled(weights) failed (%d)", (int)r); return false; }
    }
    GemmParams p = {};
    p.ctl = reinterpret_cast<const int*>(ctl); p.rows_from = rows_from;
    p.out = dst; p.bias = reinterpret_cast<const __nv_bfloat16*>(bias_bf16); p.M = M; p.N = N; p.K = K; p.out_rs = dst_rs; p.act = act; p.act_p = act_p; p.act_lo = act_lo; p.act_hi = act_hi;
    p.out_vec4 = ((reinterpret_cast<uintptr_t>(dst) & 15) == 0 && (dst_rs & 3) == 0) ? 1u : 0u;
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (act >= (uint32_t)kActs) { zg_set_error("dense gemm: unknown activation %u", act); return false; }
    g_kernel[pairs ? 1 : 0][act]<<<grid, kThreads, kSmem, st>>>(map_a, map_b, p);
    ZG_COUNT_LAUNCH();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { zg_set_error("dense gemm launch failed: %s", cudaGetErrorString(e)); return false; }
    return true;
}

static bool expert_weights_map(CUtensorMap* map, const void* w, uint32_t E, uint32_t N, uint32_t K) {
    const cuuint64_t gdim[3] = {K, N, E}, gstride[2] = {(cuuint64_t)K * 2, (cuuint64_t)N * K * 2};
    const cuuint32_t box[3] = {BK, BM, 1}, estr[3] = {1, 1, 1};
    const CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(w), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) zg_set_error("cuTensorMapEncodeTiled(expert weights) failed (%d)", (int)r);
    return r == CUDA_SUCCESS;
}
// xb: bf16 rows [rows][K] sorted by expert; w, w2: [E][N][K] bfloat16 (w2 null: out = f32 [rows][N]; otherwise out = bf16 [rows][N] of gate and up).
// d_segments: `segments` runs of rows on the device (ZgExpertSegment), those with rows first; likely_runs: how many will have some, with half a run more per expert than the rows fill.
// One matrix is taken 256 rows at a time where tiles of 128 rows would be more than the SMs: half as many take one round instead of two, and the runs' rows cross the L2 half as often.
// The op, tiles of 128 / of 256 rows: 64 tokens, two of 16 experts, ff 2048, 1024 columns (128 tiles of 128 rows) 54.9 / 55.8 us, 1280 (160) 68.7 / 63.7, 2048 87.1 / 86.4; 100
// tokens, one of 12, ff 1536, 1536 columns (144) 49.3 / 49.4, 1792 (168) 57.4 / 53.5; 1024 tokens, two of 8, ff 2048, 1024 columns (96) 91.9 / 97.6, 1792 (168) 124.3 / 118.2.  At
// several rounds either way the two differ by -3 to 7 %.  More tiles than SMs are walked by one CTA per SM (k_expert_gemm); where there are fewer, the walk's preparations
// cost (1000 tokens, one of 8 experts, 400 / 1800, 120 tiles: 47.2 us, walked 48.9).
bool zg_expert_gemm_launch(const void* w, const void* w2, uint32_t E, const void* xb, uint32_t rows, const ZgExpertSegment* d_segments, uint32_t segments, uint32_t likely_runs, void* out, uint32_t N, uint32_t K,
                           float limit, float alpha, float up_offset, cudaStream_t st) {
    if (!prepare()) return false;
    CUtensorMap map_x, map_w, map_w2;
    const cuuint64_t gdim[2] = {K, rows}, gstride[1] = {(cuuint64_t)K * 2};
    const cuuint32_t box[2] = {BK, kExpertRows}, estr[2] = {1, 1};
    const CUresult r = g_encode(&map_x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(xb), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { zg_set_error("cuTensorMapEncodeTiled(expert rows) failed (%d)", (int)r); return false; }
    if (!expert_weights_map(&map_w, w, E, N, K) || !expert_weights_map(&map_w2, w2 ? w2 : w, E, N, K)) return false;
    const ExpertParams p = {out, d_segments, N, K, segments, limit, alpha, up_offset};
    const int mode = w2 ? kExpertDual : (N + BM - 1) / BM * likely_runs > zg_sm_count() ? kExpertWide : kExpertOne;
    const uint32_t n_f = (N + (mode == kExpertWide ? 2 : 1) * BM - 1) / ((mode == kExpertWide ? 2 : 1) * BM);
    const bool loop = n_f * likely_runs > zg_sm_count();
    launch_pdl(g_expert[mode][loop], loop ? dim3(zg_sm_count()) : dim3(n_f, segments), dim3(kExpertThreads), kExpertSmem, st, map_x, map_w, map_w2, p);
    ZG_COUNT_LAUNCH();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { zg_set_error("expert gemm launch failed: %s", cudaGetErrorString(e)); return false; }
    return true;
}

bool zg_dense_gemm_batched_usable(uint32_t M, uint32_t N, uint32_t K, uint32_t act) { return M > 8 && N >= 8 && K >= 64 && K % 8 == 0 && batched_kernel(act) != nullptr; }
size_t zg_dense_gemm_batched_scratch_elems(uint32_t heads, uint32_t M, uint32_t K) { return (size_t)heads * zg_dense_gemm_scratch_elems(M, K); }
bool zg_dense_gemm_batched_launch(const void* w_bf16, const float* src, float* dst, uint32_t heads, uint32_t M, uint32_t N, uint32_t n_last, uint32_t K, uint32_t src_hs, uint32_t src_rs,
                                  uint32_t dst_hs, uint32_t dst_rs, float* scratch, cudaStream_t st, uint32_t act_last, float act_p) {
    if (!prepare()) return false;
    const uint32_t Kp = (K + BK - 1) / BK * BK, Mp = (M + BM - 1) / BM * BM;
    uint32_t* xb = reinterpret_cast<uint32_t*>(scratch);
    k_to_bf16<<<dim3((Kp / 2 + 255) / 256, Mp, heads), 256, 0, st>>>(src, src_rs, xb, Kp / 2, M, K, (const float*)nullptr, 0u, 0u, src_hs);
    ZG_COUNT_LAUNCH();
    CUtensorMap map_a, map_b;
    const cuuint32_t estr[2] = {1, 1};
    const cuuint64_t adim[2] = {Kp, (cuuint64_t)heads * Mp}, astride[1] = {(cuuint64_t)Kp * 2};
    const cuuint32_t abox[2] = {BK, BM};
    CUresult r = g_encode(&map_a, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, xb, adim, astride, abox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { zg_set_error("cuTensorMapEncodeTiled(batched rows) failed (%d)", (int)r); return false; }
    const cuuint64_t bdim[2] = {K, (cuuint64_t)(heads - 1) * N + n_last}, bstride[1] = {(cuuint64_t)K * 2};
    const cuuint32_t bbox[2] = {BK, BN};
    r = g_encode(&map_b, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(w_bf16), bdim, bstride, bbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                 CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { zg_set_error("cuTensorMapEncodeTiled(batched weights) failed (%d)", (int)r); return false; }
    GemmParams p = {};
    p.out = dst; p.M = M; p.N = N; p.K = K; p.out_rs = dst_rs; p.act = act_last; p.act_p = act_p; p.act_lo = 0; p.act_hi = 0xffffffffu;
    p.heads = heads; p.n_last = n_last; p.a_rows = Mp; p.out_hs = dst_hs;
    p.out_vec4 = ((reinterpret_cast<uintptr_t>(dst) & 15) == 0 && (dst_rs & 3) == 0 && (dst_hs & 3) == 0) ? 1u : 0u;
    GemmKernel kernel = batched_kernel(act_last);
    if (!kernel) { zg_set_error("batched dense gemm: activation %u", act_last); return false; }
    kernel<<<dim3(((N > n_last ? N : n_last) + BN - 1) / BN, Mp / BM, heads), kThreads, kSmem, st>>>(map_a, map_b, p);
    ZG_COUNT_LAUNCH();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { zg_set_error("batched dense gemm launch failed: %s", cudaGetErrorString(e)); return false; }
    return true;
}
