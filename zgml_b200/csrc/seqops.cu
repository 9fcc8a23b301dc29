// Sequence-model DeviceOps (ZG_OP_EMBED .. ZG_OP_MOE_FFN, parameter packs documented in include/zgml_cuda.h): dense
// 16-bit / f32 weights against f32 activations, affine norms with a fused residual, windowed attention with a sink over a
// key ring, short causal convolutions with a carried tail, the gated delta-rule recurrence with per-channel decay, and a
// routed mixture of experts.  Everything is accumulated in f32; a bfloat16 weight is widened exactly on load, so the two
// weight formats differ only in bytes streamed.
//
// Per-sequence state lives in external program buffers indexed by the state slot of the control buffer; the position of
// the step's first token comes from the same place, so a captured graph replays unchanged from step to step.
#include "split_tc.cuh"

#include <stdlib.h>

namespace {

// ── EMBED ─────────────────────────────────────────────────────────────────────────────────────────────────────────
template <typename WT>
__global__ void k_embed(float* __restrict__ dst, const float* __restrict__ ctl, const WT* __restrict__ table, uint32_t D, float scale,
                        const WT* __restrict__ positions, const WT* __restrict__ bigram, uint32_t buckets, uint32_t mul_prev, uint32_t mul_cur, const WT* __restrict__ dyt) {
    pdl_enter();
    const uint32_t t = blockIdx.x, c = blockIdx.y * blockDim.x + threadIdx.x;
    if (c >= D) return;
    const int id = ctl_word(ctl, ZG_CTL_IDS + t);
    float add = 0.0f;
    if (bigram) {          // a row chosen by a hash of the previous and the current token, not scaled; a sequence's first token takes the last row
        const int prev = t ? ctl_word(ctl, ZG_CTL_IDS + t - 1) : ctl_word(ctl, ZG_CTL_PREV);
        const unsigned long long b = prev < 0 ? (unsigned long long)buckets : ((unsigned long long)prev * mul_prev + (unsigned long long)id * mul_cur) % buckets;
        add = wld(bigram, (size_t)b * D + c);
    } else if (positions) {       // a learned position row, not scaled
        add = wld(positions, ((size_t)ctl_word(ctl, ZG_CTL_POS) + t) * D + c);
    }
    float x = fmaf(wld(table, (size_t)id * D + c), scale, add);
    if (dyt) x = fmaf(tanhf(wld(dyt, (size_t)2 * D) * x), wld(dyt, c), wld(dyt, (size_t)D + c));      // Dynamic Tanh: weight | bias | alpha
    dst[(size_t)t * D + c] = x;
}

// ── LINEAR, few rows (decode): one warp per output feature, the weight row streamed once for all rows ─────────────────
constexpr int kGemvRows = 8;
// PAIRS: weight rows 2n and 2n + 1 are a gate and what it multiplies, dst[., n] = act(row 2n . x) * (row 2n + 1 . x)
template <typename WT, bool PAIRS>
__global__ void k_linear_rows(float* __restrict__ dst, const float* __restrict__ src, const WT* __restrict__ W, const WT* __restrict__ bias,
                              uint32_t M, uint32_t N, uint32_t K, uint32_t src_rs, uint32_t dst_rs, SeqAct act, const float* __restrict__ ctl,
                              uint32_t slot_stride) {
    pdl_enter();
    if (ctl) src += (size_t)ctl_word(ctl, ZG_CTL_SLOT) * slot_stride;      // the rows of a per-sequence state buffer
    const uint32_t n = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (n >= N) return;
    const WT* w = W + (size_t)(PAIRS ? 2 * n : n) * K;
    float acc[kGemvRows], up[kGemvRows];
#pragma unroll
    for (int m = 0; m < kGemvRows; m++) acc[m] = up[m] = 0.0f;
    for (uint32_t k = lane; k < K; k += 32) {
        const float wv = wld(w, k), uv = PAIRS ? wld(w, (size_t)K + k) : 0.0f;
#pragma unroll
        for (int m = 0; m < kGemvRows; m++)
            if (m < (int)M) {
                const float x = src[(size_t)m * src_rs + k];
                acc[m] = fmaf(x, wv, acc[m]);
                if (PAIRS) up[m] = fmaf(x, uv, up[m]);
            }
    }
    const float b = bias && !PAIRS ? wld(bias, n) : 0.0f;
#pragma unroll
    for (int m = 0; m < kGemvRows; m++) {
        if (m < (int)M) {
            const float s = warp_sum(acc[m]), u = PAIRS ? warp_sum(up[m]) : 1.0f;
            if (lane == 0) dst[(size_t)m * dst_rs + n] = PAIRS ? seq_epilogue(s, act.kind, act.p) * u : seq_epilogue(s + b, act, n);
        }
    }
}
// The activation rows are staged once per CTA in shared memory (float4 reads, no per-weight global loads); four weight
// vectors per lane are in flight per trip.
template <typename WT, int MR, bool PAIRS>
__global__ void k_linear_rows_vec(float* __restrict__ dst, const float* __restrict__ src, const WT* __restrict__ W, const WT* __restrict__ bias,
                                  uint32_t M, uint32_t N, uint32_t K, uint32_t src_rs, uint32_t dst_rs, SeqAct act, const float* __restrict__ ctl,
                                  uint32_t slot_stride) {
    // Weights are constants of the model, so this warp's weight row is pulled toward L2 BEFORE the wait on the predecessor:
    // in a replayed graph the HBM stream of a matvec starts under the tail of the kernel that produces its input.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    {
        const uint32_t n0 = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
        if (n0 < N) {
            const char* wb = reinterpret_cast<const char*>(W + (size_t)(PAIRS ? 2 * n0 : n0) * K);
            for (size_t b = (size_t)(threadIdx.x & 31) * 128; b < (size_t)(PAIRS ? 2 : 1) * K * sizeof(WT); b += 32 * 128)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(wb + b));
        }
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    constexpr int V = WVec<WT>::n;
    extern __shared__ float xs[];                      // [M][K]
    if (ctl) src += (size_t)ctl_word(ctl, ZG_CTL_SLOT) * slot_stride;
    for (uint32_t e = threadIdx.x; e < M * K; e += blockDim.x) xs[e] = src[(size_t)(e / K) * src_rs + e % K];
    __syncthreads();
    const uint32_t n = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (n >= N) return;
    const WT* w = W + (size_t)(PAIRS ? 2 * n : n) * K;
    float acc[MR], up[MR];
#pragma unroll
    for (int m = 0; m < MR; m++) acc[m] = up[m] = 0.0f;
    auto fma_into = [&](float (&sum)[MR], const float* wv, uint32_t k) {
#pragma unroll
        for (int m = 0; m < MR; m++) {
            if (m < (int)M) {
                const float4* x = reinterpret_cast<const float4*>(xs + (size_t)m * K + k);
#pragma unroll
                for (int i = 0; i < V / 4; i++) {
                    const float4 xv = x[i];
                    sum[m] = fmaf(xv.x, wv[4 * i], fmaf(xv.y, wv[4 * i + 1], fmaf(xv.z, wv[4 * i + 2], fmaf(xv.w, wv[4 * i + 3], sum[m]))));
                }
            }
        }
    };
    auto fma_vec = [&](const float* wv, uint32_t k) { fma_into(acc, wv, k); };
    uint32_t k = lane * V;
    if constexpr (PAIRS) {                             // both rows' vectors in flight together
        const WT* wu = w + K;
        for (; k + 32 * V < K; k += 64 * V) {
            float g0[V], g1[V], u0[V], u1[V];
            wld_vec<WT>(w + k, g0);
            wld_vec<WT>(wu + k, u0);
            wld_vec<WT>(w + k + 32 * V, g1);
            wld_vec<WT>(wu + k + 32 * V, u1);
            fma_into(acc, g0, k); fma_into(up, u0, k);
            fma_into(acc, g1, k + 32 * V); fma_into(up, u1, k + 32 * V);
        }
        if (k < K) {
            float g0[V], u0[V];
            wld_vec<WT>(w + k, g0);
            wld_vec<WT>(wu + k, u0);
            fma_into(acc, g0, k); fma_into(up, u0, k);
        }
#pragma unroll
        for (int m = 0; m < MR; m++) {
            if (m < (int)M) {
                const float g = warp_sum(acc[m]), u = warp_sum(up[m]);
                if (lane == 0) dst[(size_t)m * dst_rs + n] = seq_epilogue(g, act.kind, act.p) * u;
            }
        }
    } else {
        for (; k + 96 * V < K; k += 128 * V) {
            float w0[V], w1[V], w2[V], w3[V];
            wld_vec<WT>(w + k, w0);
            wld_vec<WT>(w + k + 32 * V, w1);
            wld_vec<WT>(w + k + 64 * V, w2);
            wld_vec<WT>(w + k + 96 * V, w3);
            fma_vec(w0, k);
            fma_vec(w1, k + 32 * V);
            fma_vec(w2, k + 64 * V);
            fma_vec(w3, k + 96 * V);
        }
        for (; k + 32 * V < K; k += 64 * V) {
            float w0[V], w1[V];
            wld_vec<WT>(w + k, w0);
            wld_vec<WT>(w + k + 32 * V, w1);
            fma_vec(w0, k);
            fma_vec(w1, k + 32 * V);
        }
        if (k < K) {
            float w0[V];
            wld_vec<WT>(w + k, w0);
            fma_vec(w0, k);
        }
        const float b = bias ? wld(bias, n) : 0.0f;
#pragma unroll
        for (int m = 0; m < MR; m++) {
            if (m < (int)M) {
                const float s = warp_sum(acc[m]);
                if (lane == 0) dst[(size_t)m * dst_rs + n] = seq_epilogue(s + b, act, n);
            }
        }
    }
}

// N values in every lane -> the total of value lane % N
template <int N>
__device__ __forceinline__ float reduce_scatter(float (&v)[N], uint32_t lane) {
#pragma unroll
    for (int o = N / 2; o > 0; o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < o; i++) {
            const float keep = up ? v[i + o] : v[i], send = up ? v[i] : v[i + o];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
#pragma unroll
    for (int o = N; o < 32; o <<= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    return v[0];
}
__device__ __forceinline__ void bulk_load(float* to, const float* from, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(to)), "l"(from), "r"(bytes), "r"(bar) : "memory");
}

// ── LINEAR, few rows, weights through a ring ─────────────────────────────────────────────────────────────────────────
// One CTA per SM with a contiguous run of the weight's rows, which it brings by bulk copies through three 32 KB slots.  The first three are asked for before
// the wait on the predecessor (`early`: nothing in the program writes the weight): with two such kernels of a chain resident per SM, the HBM streams the
// next one's rows while this one's chain of norm, launch and reduction is under way.  A slot holds eight rows (of up to 4 KB pieces) per 256 threads, or
// where a row is shorter, eight rows per 32, 64 or 128 of them; a thread multiplies one 16-byte unit of each of its eight rows with the same activations.
// Shares of a row meet by shuffles and, once per 64 rows, in shared memory.
// Four gated feed-forwards of 2048 / 4096, bfloat16: one row 137 us with a warp per row and weights drawn to the L2 early, 86 now; eight rows of 1024 / 2048
// 444 us (activations that do not fit 48 KB: no staging at all) and 102.
// Activations of all rows lie in shared memory where they fit (kRingX bytes, for one and two rows whatever there is), else a segment of whole pieces of K at a
// time: then every weight row passes through once per segment, a piece of it each time, and its shares are added up in shared memory.
constexpr uint32_t kRingSlots = 3, kRingSlot = 32768, kRingPiece = 4096, kRingFlush = 64, kRingX = 65536, kRingSmem = 227 * 1024;
struct RingPlan { uint32_t ctas, lanes, segment, rows, smem; bool split; };      // segment: pieces of K whose activations are there at once; rows: whose shares are there at once
static RingPlan ring_plan(uint32_t M, uint32_t N, uint32_t K, bool pairs, uint32_t elem, uint32_t sms) {
    RingPlan r;
    const uint32_t units = K * elem / 16, pieces = (K * elem + kRingPiece - 1) / kRingPiece;
    r.ctas = std::min(sms, N);
    r.lanes = units <= 32 ? 32 : units <= 64 ? 64 : units <= 128 ? 128 : 256;
    r.split = M > 2 && (size_t)M * K * 4 > kRingX;
    r.segment = r.split ? std::min(pieces, std::max(1u, kRingX / (M * (kRingPiece / elem) * 4))) : pieces;
    r.rows = r.split ? ((N + r.ctas - 1) / r.ctas * (pairs ? 2 : 1) + 7) / 8 * 8 : 2 * kRingFlush;
    const size_t x = r.split ? (size_t)M * r.segment * (kRingPiece / elem) : (size_t)M * K, smem = kRingSlots * kRingSlot + ((size_t)r.rows * 8 * M + x) * 4 + 16 * kRingSlots + 16;
    r.smem = smem <= kRingSmem ? (uint32_t)smem : 0;                 // 0: it does not fit
    return r;
}
template <typename WT, int MR, bool PAIRS, bool SPLIT>      // SPLIT: several segments of K
__global__ void __launch_bounds__(288, MR <= 2 ? 2 : 1) k_linear_rows_ring(float* __restrict__ dst, const float* __restrict__ src, const WT* __restrict__ W, const WT* __restrict__ bias,
                                                             uint32_t M, uint32_t N, uint32_t K, uint32_t src_rs, uint32_t dst_rs, SeqAct act, const float* __restrict__ ctl,
                                                             uint32_t slot_stride, uint32_t lanes, uint32_t segment, uint32_t part_rows, uint32_t early) {
    constexpr int V = WVec<WT>::n;
    constexpr uint32_t piece_k = kRingPiece / (uint32_t)sizeof(WT);
    extern __shared__ __align__(128) unsigned char ring[];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, row_bytes = K * (uint32_t)sizeof(WT);
    // `lanes` threads (32, 64, 128, 256) share a row
    const uint32_t pieces = (row_bytes + kRingPiece - 1) / kRingPiece, group = 8 * (256 / lanes), shares = lanes >> 5, unit = tid % lanes, sub = tid / lanes;
    const uint32_t per = N / gridDim.x, more = N % gridDim.x, n0 = blockIdx.x * per + min(blockIdx.x, more), n1 = n0 + per + (blockIdx.x < more ? 1 : 0);
    const uint32_t r0 = PAIRS ? 2 * n0 : n0, rows = (PAIRS ? 2 : 1) * (n1 - n0);
    const char* w0 = reinterpret_cast<const char*>(W) + (size_t)r0 * row_bytes;
    float* part = reinterpret_cast<float*>(ring + kRingSlots * kRingSlot);      // [row][m][share], twice 64 rows or all of them
    float* xs = part + part_rows * 8 * M;                                       // [m][a segment of K]
    const uint32_t xw = SPLIT ? segment * piece_k : K;
    const uint32_t bars = smem_u32(xs + M * xw), pitch = pieces == 1 ? row_bytes : kRingPiece, failed = bars + 16 * kRingSlots;      // failed: some thread's wait gave up: the CTA's outputs are not numbers
    if (tid == 0) {
        asm volatile("st.shared.u32 [%0], %1;" ::"r"(failed), "r"(0) : "memory");
        for (uint32_t i = 0; i < kRingSlots; i++) { mbar_init(bars + 8 * i, 1); mbar_init(bars + 8 * (kRingSlots + i), 8); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    __syncthreads();
    if (warp == 8) {                                   // segment by segment of K, in a segment group by group of rows, of a group piece by piece
        if (!early) asm volatile("griddepcontrol.wait;" ::: "memory");
        uint32_t slot = 0, parity = 0, p = 0;
        bool again = false;                            // every slot has been filled once
        for (uint32_t s0 = 0; s0 < pieces; s0 = p) {
            const uint32_t s1 = SPLIT ? min(pieces, s0 + segment) : pieces;
            for (uint32_t first = 0; first < rows; first += group)
                for (p = s0; p < s1; p++) {
                    if (again && !__all_sync(0xffffffffu, mbar_wait(bars + 8 * (kRingSlots + slot), parity))) { if (lane == 0) count_timeout(); return; }
                    const uint32_t n = min(group, rows - first), bytes = min(kRingPiece, row_bytes - p * kRingPiece), bar = bars + 8 * slot;
                    unsigned char* to = ring + slot * kRingSlot;
                    const char* from = w0 + (size_t)first * row_bytes + p * kRingPiece;
                    if (lane == 0) mbar_expect_tx(bar, n * bytes);
                    __syncwarp();
                    if (pieces == 1) {
                        if (lane == 0) bulk_load(reinterpret_cast<float*>(to), reinterpret_cast<const float*>(from), n * bytes, bar);
                    } else if (lane < n) {
                        bulk_load(reinterpret_cast<float*>(to + lane * kRingPiece), reinterpret_cast<const float*>(from + (size_t)lane * row_bytes), bytes, bar);
                    }
                    if (++slot == kRingSlots) {
                        slot = 0;
                        if (again) parity ^= 1;
                        else asm volatile("griddepcontrol.wait;" ::: "memory");      // slots come free when the predecessor has completed, however long that takes: no bounded wait before
                        again = true;
                    }
                }
        }
        return;
    }
    // The first step is run through before the wait as well, over whatever the activations' place holds, its results dropped: the instructions are there
    // when the activations are (94.6 -> 91.7 us over four feed-forwards of 2048 / 4096).
    bool warm = early && MR <= 4;
    if (!warm) asm volatile("griddepcontrol.wait;" ::: "memory");
    if (ctl && !warm) src += (size_t)ctl_word(ctl, ZG_CTL_SLOT) * slot_stride;
    auto load_x = [&](uint32_t k0) {                    // K is a multiple of four; the rows of a state buffer's slot start anywhere
        const uint32_t n = min(xw, K - k0);
        const bool vec = ((reinterpret_cast<uintptr_t>(src) & 15) | (src_rs & 3)) == 0;
        for (uint32_t m = 0; m < M; m++) {
            const float* from = src + (size_t)m * src_rs + k0;
            if (vec) for (uint32_t k = 4 * tid; k < n; k += 1024) *reinterpret_cast<float4*>(xs + m * xw + k) = *reinterpret_cast<const float4*>(from + k);
            else for (uint32_t k = tid; k < n; k += 256) xs[m * xw + k] = from[k];
        }
        bar_sync(1, 256);
    };
    if (!warm) load_x(0);
    constexpr bool TWO = MR <= 2;                       // sums of even and of odd elements, by packed FMAs, where the registers allow it
    float2 acc[8][MR];
    uint32_t slot = 0, parity = 0, done = 0, half = 0;       // done: rows whose outputs are written; half: of `part`, where a flush of 64 rows reads one and the next fills the other
    auto flush = [&](uint32_t have) {
        for (uint32_t e = tid; e < (PAIRS ? have / 2 : have) * M; e += 256) {
            const uint32_t o = MR == 1 ? e : e / M, m = MR == 1 ? 0 : e % M, n = (r0 + done) / (PAIRS ? 2 : 1) + o;
            auto sum = [&](uint32_t row) {
                const float* s = part + ((size_t)(half * kRingFlush + row) * M + m) * 8;
                float t = s[0];
                for (uint32_t i = 1; i < shares; i++) t += s[i];
                return t;
            };
            if (PAIRS) dst[(size_t)m * dst_rs + n] = seq_epilogue(sum(2 * o), act.kind, act.p) * sum(2 * o + 1);
            else dst[(size_t)m * dst_rs + n] = seq_epilogue(sum(o) + (bias ? wld(bias, n) : 0.0f), act, n);
        }
        done += have;
    };
    uint32_t s0 = 0, s1 = SPLIT ? segment : pieces, p = 0, first = 0;      // the segment, the piece, the group's first row
#pragma unroll 1
    while (true) {
        if (p == s0) {
#pragma unroll
            for (int r = 0; r < 8; r++)
#pragma unroll
                for (int m = 0; m < MR; m++) acc[r][m] = make_float2(0.0f, 0.0f);
        }
        if (!mbar_wait(bars + 8 * slot, parity)) asm volatile("st.shared.u32 [%0], %1;" ::"r"(failed), "r"(1) : "memory");
        const uint32_t k = p * piece_k + unit * V;
        if (k < K) {
            const unsigned char* w = ring + slot * kRingSlot + (size_t)sub * 8 * pitch + unit * 16;
            const float* xk = xs + (SPLIT ? k - s0 * piece_k : k);
            float x[MR][V];
#pragma unroll
            for (int m = 0; m < MR; m++)
#pragma unroll
                for (int i = 0; i < V; i += 4) {
                    const float4 y = MR <= 2 || m < (int)M ? *reinterpret_cast<const float4*>(xk + m * xw + i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    x[m][i] = y.x; x[m][i + 1] = y.y; x[m][i + 2] = y.z; x[m][i + 3] = y.w;
                }
#pragma unroll
            for (int r = 0; r < 8; r++) {
                float wv[V];
                wld_vec<WT>(reinterpret_cast<const WT*>(w + r * pitch), wv);
#pragma unroll
                for (int m = 0; m < MR; m++)
#pragma unroll
                    for (int i = 0; i < V; i += 2) {
                        if (TWO) acc[r][m] = __ffma2_rn(make_float2(wv[i], wv[i + 1]), make_float2(x[m][i], x[m][i + 1]), acc[r][m]);
                        else acc[r][m].x = fmaf(wv[i + 1], x[m][i + 1], fmaf(wv[i], x[m][i], acc[r][m].x));
                    }
            }
        }
        __syncwarp();
        if (!warm && lane == 0) mbar_arrive(bars + 8 * (kRingSlots + slot));      // the slot is free
        const bool last = ++p == s1;                    // of the group's pieces in this segment
        if (last) {
            const uint32_t row = (SPLIT ? first : half * kRingFlush + first - done) + sub * 8 + (lane & 7);
#pragma unroll
            for (int m = 0; m < MR; m++) {
                if (MR > 2 && m >= (int)M) break;
                float v[8];
#pragma unroll
                for (int r = 0; r < 8; r++) v[r] = TWO ? acc[r][m].x + acc[r][m].y : acc[r][m].x;
                const float total = reduce_scatter<8>(v, lane);
                if (lane < 8) {
                    float& to = part[(row * (MR <= 2 ? MR : M) + m) * 8 + warp % shares];
                    to = SPLIT && s0 ? to + total : total;
                }
            }
        }
        if (warm) {
            warm = false;
            asm volatile("griddepcontrol.wait;" ::: "memory");
            if (ctl) src += (size_t)ctl_word(ctl, ZG_CTL_SLOT) * slot_stride;
            load_x(0);
            p = s0;
            continue;
        }
        if (++slot == kRingSlots) { slot = 0; parity ^= 1; }
        if (!last) continue;
        first += group; p = s0;
        const bool end = first >= rows;
        if (!SPLIT) {
            if (first - done >= kRingFlush || end) {
                bar_sync(1, 256);                       // the shares are there; until the next time here, nobody writes this half
                flush(min(first, rows) - done);
                half ^= 1;
            }
            if (end) break;
        } else if (end) {
            first = 0; s0 = s1; p = s1; s1 = min(pieces, s1 + segment);
            bar_sync(1, 256);                           // everyone is done with the segment's activations, or the last shares are there
            if (s0 == pieces) break;
            load_x(s0 * piece_k);
        }
    }
    if (SPLIT) flush(rows);
    uint32_t gave_up;                                  // every wait is behind the last barrier
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(gave_up) : "r"(failed) : "memory");
    if (gave_up) {
        bar_sync(1, 256);
        for (uint32_t m = 0; m < M; m++)
            for (uint32_t n = n0 + tid; n < n1; n += 256) dst[(size_t)m * dst_rs + n] = __uint_as_float(0x7fffffffu);
        if (tid == 0) count_timeout();
    }
}

// ── LINEAR, many rows (prefill), exact f32: 64 x 64 tile, 16-deep k slices, 4 x 4 outputs per thread ──────────────────
constexpr int kTM = 64, kTN = 64, kTK = 16;
// rows_from > 0: only the rows of positions the sequence holds after this step matter (rows < position + rows_from)
// PAIRS: N counts weight rows, gate and up rows in turns; columns n and n + 1 make output n / 2
template <typename WT, bool PAIRS>
__global__ void __launch_bounds__(256) k_linear_tile(float* __restrict__ dst, const float* __restrict__ src, const WT* __restrict__ W,
                                                     const WT* __restrict__ bias, uint32_t M, uint32_t N, uint32_t K, uint32_t src_rs,
                                                     uint32_t dst_rs, SeqAct act, const float* __restrict__ ctl, uint32_t slot_stride, uint32_t rows_from) {
    __shared__ float As[kTK][kTM + 4];
    __shared__ float Ws[kTK][kTN + 4];
    if (rows_from && blockIdx.y * kTM >= (uint32_t)ctl_word(ctl, ZG_CTL_POS) + rows_from) return;
    if (ctl) src += (size_t)ctl_word(ctl, ZG_CTL_SLOT) * slot_stride;
    const uint32_t m0 = blockIdx.y * kTM, n0 = blockIdx.x * kTN;
    const uint32_t tx = threadIdx.x & 15, ty = threadIdx.x >> 4;   // outputs: rows ty * 4 + i, columns tx * 4 + j
    float acc[4][4] = {};
    for (uint32_t k0 = 0; k0 < K; k0 += kTK) {
        for (uint32_t e = threadIdx.x; e < kTM * kTK; e += 256) {
            const uint32_t r = e / kTK, kk = e % kTK;
            const uint32_t m = m0 + r, k = k0 + kk;
            As[kk][r] = (m < M && k < K) ? src[(size_t)m * src_rs + k] : 0.0f;
            const uint32_t n = n0 + r;
            Ws[kk][r] = (n < N && k < K) ? wld(W, (size_t)n * K + k) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < kTK; kk++) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; i++) { a[i] = As[kk][ty * 4 + i]; b[i] = Ws[kk][tx * 4 + i]; }
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t m = m0 + ty * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; j += PAIRS ? 2 : 1) {
            const uint32_t n = n0 + tx * 4 + j;
            if (n >= N) continue;
            if (PAIRS) dst[(size_t)m * dst_rs + n / 2] = seq_epilogue(acc[i][j], act.kind, act.p) * acc[i][min(j + 1, 3)];
            else dst[(size_t)m * dst_rs + n] = seq_epilogue(acc[i][j] + (bias ? wld(bias, n) : 0.0f), act, n);
        }
    }
}

// ── NORM: one CTA per row ────────────────────────────────────────────────────────────────────────────────────────
// dst = (res +) norm(src; w) and, when a second destination is given, dst2 = norm(dst; w2) in the same launch: the norm
// that closes a sublayer (with the residual add) and the norm that opens the next one are one kernel.
constexpr int kNormCache = 16;   // values a thread keeps: rows up to 16 x blockDim are read from memory once
template <bool CACHED, typename WF>
__device__ __forceinline__ void norm_pass(float* __restrict__ out, const float* __restrict__ x, float (&v)[kNormCache], const float* __restrict__ res,
                                          const float (&rv)[kNormCache], uint32_t cols, uint32_t kind, float eps, float* sh, bool keep, WF wfn) {
    float s = 0.0f;
    if (CACHED) {
#pragma unroll
        for (int i = 0; i < kNormCache; i++) s += v[i];
    } else {
        for (uint32_t c = threadIdx.x; c < cols; c += blockDim.x) s += x[c];
    }
    const float mean = (kind & 1u) == 0 ? block_sum(s, sh) / (float)cols : 0.0f;
    float q = 0.0f;
    if (CACHED) {
#pragma unroll
        for (int i = 0; i < kNormCache; i++) {
            const uint32_t c = threadIdx.x + i * blockDim.x;
            const float d = c < cols ? v[i] - mean : 0.0f;
            q = fmaf(d, d, q);
        }
    } else {
        for (uint32_t c = threadIdx.x; c < cols; c += blockDim.x) { const float d = x[c] - mean; q = fmaf(d, d, q); }
    }
    const float inv = 1.0f / sqrtf(block_sum(q, sh) / (float)cols + eps);
    if (CACHED) {
#pragma unroll
        for (int i = 0; i < kNormCache; i++) {
            const uint32_t c = threadIdx.x + i * blockDim.x;
            if (c < cols) {
                const float y = (v[i] - mean) * inv * wfn(i, c);
                const float o = res ? rv[i] + y : y;
                out[c] = o;
                if (keep) v[i] = o;
            }
        }
    } else {
        for (uint32_t c = threadIdx.x; c < cols; c += blockDim.x) {
            const float y = (x[c] - mean) * inv * wfn(0, c);
            out[c] = res ? res[c] + y : y;
        }
    }
}
// weight as the norm applies it: stored around zero (kind bit 1) and / or carrying the gain of the product that follows (bit 2)
__device__ __forceinline__ float norm_weight(float w, uint32_t kind, float gain) {
    if (kind & 2u) w += 1.0f;
    return (kind & 4u) ? w * gain : w;
}
// kind bit 5: the weight is a single number for all columns
__device__ __forceinline__ uint32_t norm_col(uint32_t c, uint32_t kind) { return (kind & 32u) ? 0u : c; }
template <typename WT>
__global__ void k_norm(float* __restrict__ dst, const float* __restrict__ src, const WT* __restrict__ w, const float* __restrict__ res,
                       uint32_t cols, uint32_t kind, float eps, float* __restrict__ dst2, const WT* __restrict__ w2, uint32_t kind2, float gain,
                       const WT* __restrict__ shift_mix, float* __restrict__ shift_state, const float* __restrict__ ctl,
                       const WT* __restrict__ avg_coeff, uint32_t avg_terms, uint32_t avg_stride, float* __restrict__ avg_out, bool weights_first) {
    // Rows that fit the registers: norm weights that nothing in the program writes (weights_first) are read BEFORE the wait on the predecessor;
    // the row and the residual are read together right after it, so the kernel has one round of global loads, not three.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (!weights_first) asm volatile("griddepcontrol.wait;" ::: "memory");
    __shared__ float sh[32];
    const size_t row = (size_t)blockIdx.x * cols;
    const float* x = src + row;
    const bool cached = cols <= kNormCache * blockDim.x;
    float v[kNormCache], rv[kNormCache], wa[kNormCache], wb[kNormCache];
    if (cached) {
#pragma unroll
        for (int i = 0; i < kNormCache; i++) {
            const uint32_t c = threadIdx.x + i * blockDim.x;
            wa[i] = c < cols ? norm_weight(wld(w, norm_col(c, kind)), kind, gain) : 0.0f;
            wb[i] = (dst2 && c < cols) ? norm_weight(wld(w2, norm_col(c, kind2)), kind2, gain) : 0.0f;
        }
    }
    if (weights_first) asm volatile("griddepcontrol.wait;" ::: "memory");
    if (cached) {
        if (avg_terms) {   // the row to norm is a weighted sum of `avg_terms` streams (a depth average), kept in avg_out too
#pragma unroll
            for (int i = 0; i < kNormCache; i++) { v[i] = 0.0f; rv[i] = 0.0f; }
            for (uint32_t j = 0; j < avg_terms; j++) {     // one batch of independent loads per stream
                const float cj = wld(avg_coeff, j);
                const float* xj = x + (size_t)j * avg_stride;
#pragma unroll
                for (int i = 0; i < kNormCache; i++) {
                    const uint32_t c = threadIdx.x + i * blockDim.x;
                    if (c < cols) v[i] = fmaf(cj, xj[c], v[i]);
                }
            }
#pragma unroll
            for (int i = 0; i < kNormCache; i++) {
                const uint32_t c = threadIdx.x + i * blockDim.x;
                if (c < cols) avg_out[row + c] = v[i];
            }
        } else {
#pragma unroll
            for (int i = 0; i < kNormCache; i++) {
                const uint32_t c = threadIdx.x + i * blockDim.x;
                v[i] = c < cols ? x[c] : 0.0f;
                rv[i] = (res && c < cols) ? res[row + c] : 0.0f;
            }
        }
        norm_pass<true>(dst + row, x, v, res ? res + row : nullptr, rv, cols, kind, eps, sh, dst2 != nullptr, [&](int i, uint32_t) { return wa[i]; });
        if (dst2) norm_pass<true>(dst2 + row, dst + row, v, nullptr, rv, cols, kind2, eps, sh, false, [&](int i, uint32_t) { return wb[i]; });
    } else {
        if (avg_terms) {
            for (uint32_t c = threadIdx.x; c < cols; c += blockDim.x) {
                float acc = 0.0f;
                for (uint32_t j = 0; j < avg_terms; j++) acc = fmaf(wld(avg_coeff, j), x[(size_t)j * avg_stride + c], acc);
                avg_out[row + c] = acc;
            }
            __syncthreads();
            x = avg_out + row;
        }
        norm_pass<false>(dst + row, x, v, res ? res + row : nullptr, rv, cols, kind, eps, sh, false, [&](int, uint32_t c) { return norm_weight(wld(w, norm_col(c, kind)), kind, gain); });
        if (dst2) {
            __syncthreads();                           // the row just written is read back by other threads
            norm_pass<false>(dst2 + row, dst + row, v, nullptr, rv, cols, kind2, eps, sh, false, [&](int, uint32_t c) { return norm_weight(wld(w2, norm_col(c, kind2)), kind2, gain); });
        }
    }
    // Single-row steps: the token shift of the launch's last output happens here too.  Every thread revisits the columns it
    // wrote itself, so no barrier is needed; the state keeps the row as it was before the shift.
    if (shift_state) {
        float* st = shift_state + (size_t)ctl_word(ctl, ZG_CTL_SLOT) * cols;
        float* last = dst2 ? dst2 : dst;
        for (uint32_t c = threadIdx.x; c < cols; c += blockDim.x) {
            const float h = last[row + c], prev = st[c];
            st[c] = h;
            last[row + c] = fmaf(prev - h, wld(shift_mix, c), h);
        }
    }
}

// Kinds without row statistics (Dynamic Tanh; the plain residual step), their combinations with the others, and the sum of TWO
// normed sources: one CTA per row.  dst = (res +) f(src) (+ f_b(src_b)) and, with dst2, dst2 = f2(dst): the residual step that
// closes a sublayer and the Dynamic Tanh that opens the next are one launch.  Rows of up to kNormCache x blockDim values live in
// registers: weights and biases are constants of the model and are read BEFORE the wait on the predecessor, the row, its
// residual and the second source together right after it.  Wider rows are walked from memory.
template <typename WT>
__device__ __forceinline__ float norm_any_value(float x, float mean, float inv, float w, float aux, uint32_t kind, float gain, float alpha) {
    const float g = (kind & 4u) ? gain : 1.0f;
    if (kind & 16u) return x * g;
    if (kind & 8u) return fmaf(tanhf(alpha * x), w, aux) * g;
    return (x - mean) * inv * ((kind & 2u) ? w + 1.0f : w) * g;
}
template <typename WT>
__device__ void norm_any_pass(float* out, const float* x, const float* res, const WT* __restrict__ w, uint32_t cols, uint32_t kind, float eps, float gain,
                              float* sh, const float* xb, const WT* __restrict__ wb) {
    float mean = 0.0f, inv = 1.0f, mean_b = 0.0f, inv_b = 1.0f;
    if (!(kind & 24u)) {
        if (!(kind & 1u)) {
            float sum = 0.0f, sum_b = 0.0f;
            for (uint32_t c = threadIdx.x; c < cols; c += blockDim.x) { sum += x[c]; if (xb) sum_b += xb[c]; }
            mean = block_sum(sum, sh) / (float)cols;
            if (xb) mean_b = block_sum(sum_b, sh) / (float)cols;
        }
        float q = 0.0f, qb = 0.0f;
        for (uint32_t c = threadIdx.x; c < cols; c += blockDim.x) {
            const float d = x[c] - mean; q = fmaf(d, d, q);
            if (xb) { const float e = xb[c] - mean_b; qb = fmaf(e, e, qb); }
        }
        inv = 1.0f / sqrtf(block_sum(q, sh) / (float)cols + eps);
        if (xb) inv_b = 1.0f / sqrtf(block_sum(qb, sh) / (float)cols + eps);
    }
    const float alpha = (kind & 8u) ? wld(w, (size_t)2 * cols) : 0.0f;
    for (uint32_t c = threadIdx.x; c < cols; c += blockDim.x) {
        float y = norm_any_value<WT>(x[c], mean, inv, (kind & 16u) ? 0.0f : wld(w, norm_col(c, kind)), (kind & 8u) ? wld(w, (size_t)cols + c) : 0.0f, kind, gain, alpha);
        if (xb) y += norm_any_value<WT>(xb[c], mean_b, inv_b, wld(wb, norm_col(c, kind)), 0.0f, kind, gain, 0.0f);
        out[c] = res ? res[c] + y : y;
    }
}
// with an outer norm (w_o) the sum itself is normed once more before it joins the residual.  Every pass touches a column from
// the same thread, so the second one may run in place.
template <typename WT>
__device__ void norm_any_sum(float* out, const float* x, const float* res, const WT* __restrict__ w, uint32_t cols, uint32_t kind, float eps, float gain, float* sh,
                             const float* xb, const WT* __restrict__ wb, uint32_t kind_o, const WT* __restrict__ w_o) {
    norm_any_pass(out, x, w_o ? (const float*)nullptr : res, w, cols, kind, eps, gain, sh, xb, wb);
    if (w_o) norm_any_pass(out, out, res, w_o, cols, kind_o, eps, gain, sh, (const float*)nullptr, (const WT*)nullptr);
}
// more rows than fit at once in registers (and narrow ones): what counts is how many rows are resident per SM, so nothing is kept in registers
template <typename WT>
__global__ void __launch_bounds__(256) k_norm_any_rows(float* dst, const float* src, const WT* __restrict__ w, const float* res, uint32_t cols, uint32_t kind, float eps,
                                                       float* dst2, const WT* __restrict__ w2, uint32_t kind2, float gain, const float* src_b, const WT* __restrict__ w_b,
                                                       uint32_t kind_o, const WT* __restrict__ w_o) {
    pdl_enter();
    __shared__ float sh[32];
    const size_t row = (size_t)blockIdx.x * cols;
    norm_any_sum(dst + row, src + row, res ? res + row : nullptr, w, cols, kind, eps, gain, sh, src_b ? src_b + row : nullptr, w_b, kind_o, w_o);
    if (dst2) {
        __syncthreads();                                   // the row just written is read back by other threads
        norm_any_pass(dst2 + row, dst + row, (const float*)nullptr, w2, cols, kind2, eps, gain, sh, (const float*)nullptr, (const WT*)nullptr);
    }
}
// A thread's share of a weight, or of one value for all columns (kind bit 5).  The column is clamped instead of tested and whether the
// weight is there at all is decided once, so that all loads are in flight before the first is widened; shares past the row are unused.
template <typename WT, int kKeep>
__device__ __forceinline__ void norm_any_weights(float (&out)[kKeep], const WT* __restrict__ w, bool have, uint32_t cols, uint32_t kind) {
    if (!have) {
#pragma unroll
        for (int i = 0; i < kKeep; i++) out[i] = 0.0f;
        return;
    }
    WT raw[kKeep];
#pragma unroll
    for (int i = 0; i < kKeep; i++) raw[i] = w[norm_col(min(threadIdx.x + i * blockDim.x, cols - 1), kind)];
#pragma unroll
    for (int i = 0; i < kKeep; i++) out[i] = wld(raw + i, 0);
}
template <typename WT, int kKeep, int kThreads>          // a row of up to kKeep x kThreads values lives in registers (fewer kept values, more CTAs per SM)
__global__ void __launch_bounds__(kThreads) k_norm_any(float* dst, const float* src, const WT* __restrict__ w, const float* res, uint32_t cols, uint32_t kind, float eps,
                                                  float* dst2, const WT* __restrict__ w2, uint32_t kind2, float gain, const float* src_b, const WT* __restrict__ w_b,
                                                       uint32_t kind_o, const WT* __restrict__ w_o, bool weights_first) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    __shared__ float sh[kThreads > 512 ? kThreads / 16 : 32];      // of a warp: one sum, or the two sources'
    const size_t row = (size_t)blockIdx.x * cols;
    if (cols > kKeep * kThreads) {                  // rows too wide for the registers
        asm volatile("griddepcontrol.wait;" ::: "memory");
        norm_any_sum(dst + row, src + row, res ? res + row : nullptr, w, cols, kind, eps, gain, sh, src_b ? src_b + row : nullptr, w_b, kind_o, w_o);
        if (dst2) {
            __syncthreads();                               // the row just written is read back by other threads
            norm_any_pass(dst2 + row, dst + row, (const float*)nullptr, w2, cols, kind2, eps, gain, sh, (const float*)nullptr, (const WT*)nullptr);
        }
        return;
    }
    if (!weights_first) asm volatile("griddepcontrol.wait;" ::: "memory");
    float v[kKeep], wa[kKeep], aux[kKeep], wc[kKeep], bc[kKeep], wo[kKeep];   // aux: the bias of a Dynamic Tanh, or the second source's weight
    norm_any_weights<WT, kKeep>(wa, w, !(kind & 16u), cols, kind);
    norm_any_weights<WT, kKeep>(aux, (kind & 8u) ? w + cols : w_b, (kind & 8u) || src_b, cols, kind);
    norm_any_weights<WT, kKeep>(wc, w2, dst2 && !(kind2 & 16u), cols, kind2);
    norm_any_weights<WT, kKeep>(wo, w_o, w_o != nullptr, cols, kind_o);
    norm_any_weights<WT, kKeep>(bc, w2 + cols, dst2 && (kind2 & 8u), cols, kind2);
    const float alpha = (kind & 8u) ? wld(w, (size_t)2 * cols) : 0.0f, alpha2 = (dst2 && (kind2 & 8u)) ? wld(w2, (size_t)2 * cols) : 0.0f;
    if (weights_first) asm volatile("griddepcontrol.wait;" ::: "memory");
    float rv[kKeep], vb[kKeep];
#pragma unroll
    for (int i = 0; i < kKeep; i++) {
        const uint32_t c = threadIdx.x + i * blockDim.x;
        v[i] = c < cols ? src[row + c] : 0.0f;
        rv[i] = (res && c < cols) ? res[row + c] : 0.0f;
        vb[i] = (src_b && c < cols) ? src_b[row + c] : 0.0f;
    }
    auto stats = [&](const float (&val)[kKeep], uint32_t k, float& mean, float& inv) {
        mean = 0.0f; inv = 1.0f;
        if (k & 24u) return;
        if (!(k & 1u)) {
            float sum = 0.0f;
#pragma unroll
            for (int i = 0; i < kKeep; i++) sum += val[i];
            mean = block_sum(sum, sh) / (float)cols;
        }
        float q = 0.0f;
#pragma unroll
        for (int i = 0; i < kKeep; i++) {
            const float d = threadIdx.x + i * blockDim.x < cols ? val[i] - mean : 0.0f;
            q = fmaf(d, d, q);
        }
        inv = 1.0f / sqrtf(block_sum(q, sh) / (float)cols + eps);
    };
    float mean, inv, mean_b = 0.0f, inv_b = 1.0f;
    if (src_b && (kind & 1u)) {                     // both sources' root mean squares in one reduction
        float q = 0.0f, qb = 0.0f;
#pragma unroll
        for (int i = 0; i < kKeep; i++) { q = fmaf(v[i], v[i], q); qb = fmaf(vb[i], vb[i], qb); }
        const float2 s2 = block_sum2<kThreads>(q, qb, sh);
        inv = 1.0f / sqrtf(s2.x / (float)cols + eps); inv_b = 1.0f / sqrtf(s2.y / (float)cols + eps);
        mean = 0.0f;
    } else {
        stats(v, kind, mean, inv);
        if (src_b) stats(vb, kind, mean_b, inv_b);
    }
#pragma unroll
    for (int i = 0; i < kKeep; i++) {
        const uint32_t c = threadIdx.x + i * blockDim.x;
        if (c >= cols) { v[i] = 0.0f; continue; }       // columns past the row stay zero (a layer norm would shift them)
        float y = norm_any_value<WT>(v[i], mean, inv, wa[i], aux[i], kind, gain, alpha);
        if (src_b) y += norm_any_value<WT>(vb[i], mean_b, inv_b, aux[i], 0.0f, kind, gain, 0.0f);
        if (w_o) { v[i] = y; continue; }
        v[i] = res ? rv[i] + y : y;
        if (c < cols) dst[row + c] = v[i];
    }
    if (w_o) {                                      // the sum is normed once more before it joins the residual
        stats(v, kind_o, mean, inv);
#pragma unroll
        for (int i = 0; i < kKeep; i++) {
            const uint32_t c = threadIdx.x + i * blockDim.x;
            const float y = norm_any_value<WT>(v[i], mean, inv, wo[i], 0.0f, kind_o, gain, 0.0f);
            v[i] = res ? rv[i] + y : y;
            if (c < cols) dst[row + c] = v[i];
        }
    }
    if (!dst2) return;
    stats(v, kind2, mean, inv);
#pragma unroll
    for (int i = 0; i < kKeep; i++) {
        const uint32_t c = threadIdx.x + i * blockDim.x;
        if (c < cols) dst2[row + c] = norm_any_value<WT>(v[i], mean, inv, wc[i], bc[i], kind2, gain, alpha2);
    }
}

// ── WINDOW_ATTENTION ─────────────────────────────────────────────────────────────────────────────────────────────
__global__ void k_ring_append(float* __restrict__ ring, const float* __restrict__ proj, const float* __restrict__ ctl, uint32_t k_off,
                              uint32_t proj_rs, uint32_t width, uint32_t R) {
    pdl_enter();
    const uint32_t t = blockIdx.x;
    const uint32_t pos = (uint32_t)ctl_word(ctl, ZG_CTL_POS) + t, slot = (uint32_t)ctl_word(ctl, ZG_CTL_SLOT);
    float* row = ring + ((size_t)slot * R + pos % R) * width;
    const float* k = proj + (size_t)t * proj_rs + k_off;
    for (uint32_t c = threadIdx.x; c < width; c += blockDim.x) row[c] = k[c];
}
constexpr int kAttnMaxDim = 256;   // 8 channels per lane
// one warp per (token, head): 32 keys at a time, lane = key for the scores, lane = channel for the weighted sum
__global__ void k_window_attention(float* __restrict__ dst, const float* __restrict__ proj, const float* __restrict__ ring,
                                   const float* __restrict__ bias, const float* __restrict__ ctl, uint32_t T, uint32_t H, uint32_t G,
                                   uint32_t dim, uint32_t proj_rs, uint32_t q_off, uint32_t g_off, uint32_t window, uint32_t R,
                                   float scale, float cap) {
    pdl_enter();
    extern __shared__ float sq[];                      // [warps][dim]
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const uint32_t item = blockIdx.x * nw + warp;
    if (item >= T * H) return;
    const uint32_t t = item / H, h = item % H, kv = h / (H / G);
    const uint32_t pos0 = (uint32_t)ctl_word(ctl, ZG_CTL_POS), slot = (uint32_t)ctl_word(ctl, ZG_CTL_SLOT);
    const uint32_t p = pos0 + t;
    const uint32_t lo = p + 1 >= window ? p + 1 - window : 0;
    float* q = sq + warp * dim;
    const float* qrow = proj + (size_t)t * proj_rs + q_off + (size_t)h * dim;
    for (uint32_t c = lane; c < dim; c += 32) q[c] = qrow[c];
    __syncwarp();
    const size_t width = (size_t)G * dim;
    const float* base = ring + (size_t)slot * R * width + (size_t)kv * dim;
    float m = 0.0f, l = 1.0f;                          // the sink: score 0, weight exp(0 - m), no value
    float acc[kAttnMaxDim / 32];
#pragma unroll
    for (int i = 0; i < kAttnMaxDim / 32; i++) acc[i] = 0.0f;
    for (uint32_t j0 = lo; j0 <= p; j0 += 32) {
        const uint32_t j = j0 + lane;
        float s = -INFINITY;
        if (j <= p) {
            const float* k = base + (size_t)(j % R) * width;
            float d = 0.0f;
            for (uint32_t c = 0; c < dim; c++) d = fmaf(q[c], k[c], d);
            s = d * scale;
            if (cap > 0.0f) s = cap * tanhf(s / cap);
            s += bias[(size_t)(p - j) * H + h];
        }
        const float m_new = fmaxf(m, warp_max(s));
        const float corr = expf(m - m_new);
        const float e = j <= p ? expf(s - m_new) : 0.0f;
        l = l * corr + warp_sum(e);
        m = m_new;
        const uint32_t cnt = min(32u, p - j0 + 1);
#pragma unroll
        for (int i = 0; i < kAttnMaxDim / 32; i++) acc[i] *= corr;
        for (uint32_t jj = 0; jj < cnt; jj++) {
            const float pj = __shfl_sync(0xffffffffu, e, jj);
            const float* k = base + (size_t)((j0 + jj) % R) * width;
#pragma unroll
            for (int i = 0; i < kAttnMaxDim / 32; i++) {
                const uint32_t c = lane + 32 * i;
                if (c < dim) acc[i] = fmaf(pj, k[c], acc[i]);
            }
        }
    }
    const float inv = 1.0f / l;
    const float* grow = proj + (size_t)t * proj_rs + g_off + (size_t)h * dim;
    float* out = dst + ((size_t)t * H + h) * dim;
#pragma unroll
    for (int i = 0; i < kAttnMaxDim / 32; i++) {
        const uint32_t c = lane + 32 * i;
        if (c < dim) out[c] = acc[i] * inv * sigmoidf_(grow[c]);
    }
}

// The kernel above is the fallback for head sizes that are not a multiple of 4.  This one: one CTA per (token, head), its
// warps split the window; inside a warp LK lanes share a key (each holds 4 * CH channels of it as float4s, so a key row is
// one coalesced read that serves the score AND — keys being the values — the weighted sum), 32 / LK keys per trip.  Every
// lane group keeps its own running (max, sum, accumulator); groups and warps are merged at the end, where the sink joins.
template <int CH>
__global__ void k_window_attention_v(float* __restrict__ dst, const float* __restrict__ proj, const float* __restrict__ ring,
                                     const float* __restrict__ bias, const float* __restrict__ ctl, uint32_t H, uint32_t G, uint32_t dim,
                                     uint32_t LK, uint32_t proj_rs, uint32_t q_off, uint32_t g_off, uint32_t window, uint32_t R, float scale,
                                     float cap, float* __restrict__ part) {
    pdl_enter();
    extern __shared__ float sm[];                      // [warps][4 + dim]: max, sum, two pad words (float4 alignment), accumulator
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const uint32_t t = blockIdx.x / H, h = blockIdx.x % H, kv = h / (H / G);
    const uint32_t pos0 = (uint32_t)ctl_word(ctl, ZG_CTL_POS), slot = (uint32_t)ctl_word(ctl, ZG_CTL_SLOT);
    const uint32_t p = pos0 + t;
    const uint32_t lo = p + 1 >= window ? p + 1 - window : 0;
    const uint32_t KP = 32 / LK, sub = lane % LK, ks = lane / LK;
    const float* qrow = proj + (size_t)t * proj_rs + q_off + (size_t)h * dim;
    float4 q[CH], acc[CH];
    bool valid[CH];
#pragma unroll
    for (int c = 0; c < CH; c++) {
        const uint32_t ch = (c * LK + sub) * 4;
        valid[c] = ch < dim;
        q[c] = valid[c] ? *reinterpret_cast<const float4*>(qrow + ch) : make_float4(0, 0, 0, 0);
        acc[c] = make_float4(0, 0, 0, 0);
    }
    const size_t width = (size_t)G * dim;
    const float* base = ring + (size_t)slot * R * width + (size_t)kv * dim;
    // gridDim.y CTAs split the window (decode: few (token, head) pairs, long windows), the warps of a CTA split its share
    const uint32_t n_keys = p - lo + 1;
    const uint32_t per_cta = (n_keys + gridDim.y - 1) / gridDim.y;
    const uint32_t c_begin = lo + blockIdx.y * per_cta, c_end = min(p + 1, c_begin + per_cta);
    const uint32_t per = ((c_end > c_begin ? c_end - c_begin : 0) + nw - 1) / nw;
    const uint32_t j_begin = c_begin + warp * per, j_end = min(c_end, j_begin + per);   // this warp's keys [j_begin, j_end)
    float m = -INFINITY, l = 0.0f;
    constexpr int U = 4;                               // keys in flight per lane group: their loads are issued together
    for (uint32_t j0 = j_begin; j0 < j_end; j0 += KP * U) {
        float4 kvv[U][CH];
        float d[U], bj[U];                             // the distance biases travel with the keys: no load inside the serial softmax update
        bool on[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const uint32_t j = j0 + u * KP + ks;
            on[u] = j < j_end;
            bj[u] = on[u] ? bias[(size_t)(p - j) * H + h] : 0.0f;
            const float* k = base + (size_t)(j % R) * width;
#pragma unroll
            for (int c = 0; c < CH; c++)
                kvv[u][c] = (on[u] && valid[c]) ? *reinterpret_cast<const float4*>(k + (c * LK + sub) * 4) : make_float4(0, 0, 0, 0);
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            d[u] = 0.0f;
#pragma unroll
            for (int c = 0; c < CH; c++)
                d[u] = fmaf(q[c].x, kvv[u][c].x, fmaf(q[c].y, kvv[u][c].y, fmaf(q[c].z, kvv[u][c].z, fmaf(q[c].w, kvv[u][c].w, d[u]))));
        }
        for (uint32_t o = LK >> 1; o > 0; o >>= 1) {
#pragma unroll
            for (int u = 0; u < U; u++) d[u] += __shfl_xor_sync(0xffffffffu, d[u], o);
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (!on[u]) continue;
            float sc = d[u] * scale;
            if (cap > 0.0f) sc = cap * tanhf(sc / cap);
            sc += bj[u];
            if (sc > m) {
                const float corr = expf(m - sc);        // exp(-inf) = 0 on the first key
                l *= corr;
#pragma unroll
                for (int c = 0; c < CH; c++) { acc[c].x *= corr; acc[c].y *= corr; acc[c].z *= corr; acc[c].w *= corr; }
                m = sc;
            }
            const float pj = expf(sc - m);
            l += pj;
#pragma unroll
            for (int c = 0; c < CH; c++) {
                acc[c].x = fmaf(pj, kvv[u][c].x, acc[c].x); acc[c].y = fmaf(pj, kvv[u][c].y, acc[c].y);
                acc[c].z = fmaf(pj, kvv[u][c].z, acc[c].z); acc[c].w = fmaf(pj, kvv[u][c].w, acc[c].w);
            }
        }
    }
    // merge the key slots of the warp (lanes that differ in lane / LK)
    for (uint32_t o = LK; o < 32; o <<= 1) {
        const float m2 = __shfl_xor_sync(0xffffffffu, m, o), l2 = __shfl_xor_sync(0xffffffffu, l, o);
        const float M = fmaxf(m, m2);
        const float w1 = m == -INFINITY ? 0.0f : expf(m - M), w2 = m2 == -INFINITY ? 0.0f : expf(m2 - M);
        l = l * w1 + l2 * w2;
#pragma unroll
        for (int c = 0; c < CH; c++) {
            acc[c].x = acc[c].x * w1 + __shfl_xor_sync(0xffffffffu, acc[c].x, o) * w2;
            acc[c].y = acc[c].y * w1 + __shfl_xor_sync(0xffffffffu, acc[c].y, o) * w2;
            acc[c].z = acc[c].z * w1 + __shfl_xor_sync(0xffffffffu, acc[c].z, o) * w2;
            acc[c].w = acc[c].w * w1 + __shfl_xor_sync(0xffffffffu, acc[c].w, o) * w2;
        }
        m = M;
    }
    float* mine = sm + warp * (4 + dim);
    if (lane < LK) {
        if (sub == 0) { mine[0] = m; mine[1] = l; }
#pragma unroll
        for (int c = 0; c < CH; c++)
            if (valid[c]) *reinterpret_cast<float4*>(mine + 4 + (c * LK + sub) * 4) = acc[c];
    }
    __syncthreads();
    // merge the warps
    float M = -INFINITY;
    for (uint32_t w = 0; w < nw; w++) M = fmaxf(M, sm[w * (4 + dim)]);
    float L = 0.0f;
    for (uint32_t w = 0; w < nw; w++) { const float mw = sm[w * (4 + dim)]; if (mw != -INFINITY) L += sm[w * (4 + dim) + 1] * expf(mw - M); }
    const float* grow = proj + (size_t)t * proj_rs + g_off + (size_t)h * dim;
    float* out = dst + ((size_t)t * H + h) * dim;
    float* mine_part = part ? part + ((size_t)blockIdx.x * gridDim.y + blockIdx.y) * (4 + dim) : nullptr;
    // the sink (score 0, no value) joins the denominator where the last merge happens
    const float Ms = fmaxf(M, 0.0f);
    const float wk = M == -INFINITY ? 0.0f : expf(M - Ms);
    const float inv = 1.0f / (expf(-Ms) + L * wk);
    if (mine_part && threadIdx.x == 0) { mine_part[0] = M; mine_part[1] = L; }
    for (uint32_t c = threadIdx.x; c < dim; c += blockDim.x) {
        float a = 0.0f;
        for (uint32_t w = 0; w < nw; w++) { const float mw = sm[w * (4 + dim)]; if (mw != -INFINITY) a = fmaf(sm[w * (4 + dim) + 4 + c], expf(mw - M), a); }
        if (mine_part) mine_part[4 + c] = a;
        else out[c] = a * wk * inv * sigmoidf_(grow[c]);
    }
}
// merge of the window shares of k_window_attention_v: one CTA per (token, head)
__global__ void k_window_attention_merge(float* __restrict__ dst, const float* __restrict__ proj, const float* __restrict__ part, uint32_t H, uint32_t dim,
                                         uint32_t S, uint32_t proj_rs, uint32_t g_off) {
    pdl_enter();
    const uint32_t t = blockIdx.x / H, h = blockIdx.x % H;
    const float* P = part + (size_t)blockIdx.x * S * (4 + dim);
    float M = 0.0f;                                    // the sink's score
    for (uint32_t i = 0; i < S; i++) M = fmaxf(M, P[i * (4 + dim)]);
    float L = expf(-M);
    for (uint32_t i = 0; i < S; i++) { const float mi = P[i * (4 + dim)]; if (mi != -INFINITY) L += P[i * (4 + dim) + 1] * expf(mi - M); }
    const float inv = 1.0f / L;
    const float* grow = proj + (size_t)t * proj_rs + g_off + (size_t)h * dim;
    for (uint32_t c = threadIdx.x; c < dim; c += blockDim.x) {
        float a = 0.0f;
        for (uint32_t i = 0; i < S; i++) { const float mi = P[i * (4 + dim)]; if (mi != -INFINITY) a = fmaf(P[i * (4 + dim) + 4 + c], expf(mi - M), a); }
        dst[((size_t)t * H + h) * dim + c] = a * inv * sigmoidf_(grow[c]);
    }
}

// Prefill form of WINDOW_ATTENTION (16 or more tokens, head size up to 128): flash tiling in f32, as the framework's causal
// prefill attention does.  One CTA owns 64 consecutive queries of one head and walks the keys its window reaches in tiles
// of 64 ring rows.  The key tile in shared memory serves the scores AND, keys being the values, the weighted sum.  Thread
// (ty, tx) of 16 x 16 holds queries 4 ty .. 4 ty + 3 against keys tx + 16 c (conflict-free float4 reads of padded key rows);
// the row statistics of the running softmax are shared by the 16 threads of a row through half-warp shuffles; the
// probabilities pass through shared memory; outputs tx + 16 c of the four rows accumulate in registers.  The distance
// biases a tile can meet (127 distances) are staged once per tile, -inf standing for "outside the window or the future".
// The sink joins the denominator at the end, then the output gate.  DH = 16 OC covers the head; channels past dim are zero.
constexpr int kWaBQ = 64, kWaBK = 64, kWaThreads = 256, kWaTiledMinTokens = 16;
template <int OC>
__global__ void __launch_bounds__(kWaThreads, 2)
k_window_attention_tiled(float* __restrict__ dst, const float* __restrict__ proj, const float* __restrict__ ring, const float* __restrict__ bias,
                         const float* __restrict__ ctl, uint32_t T, uint32_t H, uint32_t G, uint32_t dim, uint32_t proj_rs, uint32_t q_off,
                         uint32_t g_off, uint32_t window, uint32_t R, float scale, float cap, uint32_t n_sm) {
    pdl_enter();
    constexpr int DH = 16 * OC, KP = DH + 4, PP = kWaBK + 4;
    extern __shared__ __align__(16) float sm[];
    float* Qs = sm;                                    // [64][DH]
    float* Ks = Qs + kWaBQ * DH;                       // [64][DH + 4]
    float* Ps = Ks + kWaBK * KP;                       // [64][64 + 4]
    float* Bs = Ps + kWaBQ * PP;                       // [128]
    // A later query tile walks more key tiles.  Blocks are ranked heaviest first (the block scheduler hands them out in index
    // order); when the whole grid is resident at once, two CTAs per SM, the second CTA of every SM is taken from the light
    // end instead, so that each SM's pair carries about the same number of key tiles.
    uint32_t rank = blockIdx.x;
    if (gridDim.x <= 2 * n_sm && rank >= n_sm) rank = gridDim.x - 1 - (rank - n_sm);
    const uint32_t n_tiles = (T + kWaBQ - 1) / kWaBQ;
    const uint32_t h = rank % H, kv = h / (H / G), t0 = (n_tiles - 1 - rank / H) * kWaBQ;
    const uint32_t tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const uint32_t pos0 = (uint32_t)ctl_word(ctl, ZG_CTL_POS), slot = (uint32_t)ctl_word(ctl, ZG_CTL_SLOT);
    const uint32_t nq = min((uint32_t)kWaBQ, T - t0);
    const uint32_t p_first = pos0 + t0, p_last = p_first + nq - 1;
    const uint32_t lo = p_first + 1 >= window ? p_first + 1 - window : 0;
    const size_t width = (size_t)G * dim;
    const float* base = ring + (size_t)slot * R * width + (size_t)kv * dim;
    for (uint32_t i = tid; i < kWaBQ * (DH / 4); i += kWaThreads) {
        const uint32_t r = i / (DH / 4), c4 = i % (DH / 4);
        float4 val = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < nq && 4 * c4 < dim) val = *reinterpret_cast<const float4*>(proj + (size_t)(t0 + r) * proj_rs + q_off + (size_t)h * dim + 4 * c4);
        *reinterpret_cast<float4*>(Qs + r * DH + 4 * c4) = val;
    }
    float o[4][OC], m_run[4], l_run[4];
#pragma unroll
    for (int r = 0; r < 4; r++) {
        m_run[r] = -INFINITY; l_run[r] = 0.0f;
#pragma unroll
        for (int c = 0; c < OC; c++) o[r][c] = 0.0f;
    }
    for (uint32_t s0 = lo; s0 <= p_last; s0 += kWaBK) {
        __syncthreads();                               // the previous tile's readers of Ks / Ps / Bs are done
        for (uint32_t i = tid; i < kWaBK * (DH / 4); i += kWaThreads) {
            const uint32_t r = i / (DH / 4), c4 = i % (DH / 4);
            float4 val = make_float4(0.f, 0.f, 0.f, 0.f);
            if (s0 + r <= p_last && 4 * c4 < dim) val = *reinterpret_cast<const float4*>(base + (size_t)((s0 + r) % R) * width + 4 * c4);
            *reinterpret_cast<float4*>(Ks + r * KP + 4 * c4) = val;
        }
        if (tid < 2 * kWaBK - 1) {                     // distance of (query row a, key column b) = p_first - s0 + a - b
            const int d = (int)p_first - (int)s0 - (kWaBK - 1) + (int)tid;
            Bs[tid] = (d >= 0 && d < (int)window) ? bias[(size_t)d * H + h] : -INFINITY;
        }
        __syncthreads();
        float sc[4][4];
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int c = 0; c < 4; c++) sc[r][c] = 0.0f;
#pragma unroll 2
        for (int d = 0; d < DH; d += 4) {
            float4 qa[4], ka[4];
#pragma unroll
            for (int r = 0; r < 4; r++) qa[r] = *reinterpret_cast<const float4*>(Qs + (4 * ty + r) * DH + d);
#pragma unroll
            for (int c = 0; c < 4; c++) ka[c] = *reinterpret_cast<const float4*>(Ks + (tx + 16 * c) * KP + d);
#pragma unroll
            for (int r = 0; r < 4; r++)
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    sc[r][c] = fmaf(qa[r].x, ka[c].x, sc[r][c]); sc[r][c] = fmaf(qa[r].y, ka[c].y, sc[r][c]);
                    sc[r][c] = fmaf(qa[r].z, ka[c].z, sc[r][c]); sc[r][c] = fmaf(qa[r].w, ka[c].w, sc[r][c]);
                }
        }
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const uint32_t a = 4 * ty + r;
            float rmax = -INFINITY;
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const float b = Bs[a + (kWaBK - 1) - (tx + 16 * c)];
                float sv = -INFINITY;
                if (a < nq && b != -INFINITY) {
                    sv = sc[r][c] * scale;
                    if (cap > 0.0f) sv = cap * tanhf(sv / cap);
                    sv += b;
                }
                sc[r][c] = sv;
                rmax = fmaxf(rmax, sv);
            }
#pragma unroll
            for (int off = 8; off > 0; off >>= 1) rmax = fmaxf(rmax, __shfl_xor_sync(0xffffffffu, rmax, off));
            const float new_m = fmaxf(m_run[r], rmax);
            const float alpha = m_run[r] == -INFINITY ? (new_m == -INFINITY ? 1.0f : 0.0f) : expf(m_run[r] - new_m);
            float rsum = 0.0f;
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const float pv = sc[r][c] == -INFINITY ? 0.0f : expf(sc[r][c] - new_m);
                Ps[a * PP + tx + 16 * c] = pv;
                rsum += pv;
            }
#pragma unroll
            for (int off = 8; off > 0; off >>= 1) rsum += __shfl_xor_sync(0xffffffffu, rsum, off);
            l_run[r] = l_run[r] * alpha + rsum;
            m_run[r] = new_m;
#pragma unroll
            for (int c = 0; c < OC; c++) o[r][c] *= alpha;
        }
        __syncthreads();
#pragma unroll 4
        for (int j = 0; j < kWaBK; j++) {
            float pj[4], vj[OC];
#pragma unroll
            for (int r = 0; r < 4; r++) pj[r] = Ps[(4 * ty + r) * PP + j];
#pragma unroll
            for (int c = 0; c < OC; c++) vj[c] = Ks[j * KP + tx + 16 * c];
#pragma unroll
            for (int r = 0; r < 4; r++)
#pragma unroll
                for (int c = 0; c < OC; c++) o[r][c] = fmaf(pj[r], vj[c], o[r][c]);
        }
    }
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const uint32_t a = 4 * ty + r;
        if (a >= nq) continue;
        // every query sees itself, so m_run is finite; the sink (score 0, no value) joins the denominator here
        const float Ms = fmaxf(m_run[r], 0.0f);
        const float wk = expf(m_run[r] - Ms);
        const float inv = wk / (expf(-Ms) + l_run[r] * wk);
        const float* grow = proj + (size_t)(t0 + a) * proj_rs + g_off + (size_t)h * dim;
        float* out = dst + ((size_t)(t0 + a) * H + h) * dim;
#pragma unroll
        for (int c = 0; c < OC; c++) {
            const uint32_t col = tx + 16 * c;
            if (col < dim) out[col] = o[r][c] * inv * sigmoidf_(grow[col]);
        }
    }
}
template <int OC>
static void launch_window_attention_tiled(const ZgSeqOp& s, float* const* bufs, cudaStream_t st) {
    constexpr int DH = 16 * OC;
    const size_t smem = ((size_t)kWaBQ * DH + (size_t)kWaBK * (DH + 4) + (size_t)kWaBQ * (kWaBK + 4) + 2 * kWaBK) * sizeof(float);
    static bool once = false;
    if (!once) { cudaFuncSetAttribute(k_window_attention_tiled<OC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); once = true; }
    static int n_sm = 0;
    if (!n_sm) { int dev = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev); if (n_sm <= 0) n_sm = 1; }
    launch_pdl(k_window_attention_tiled<OC>, dim3(((s.n[0] + kWaBQ - 1) / kWaBQ) * s.n[1]), dim3(kWaThreads), smem, st, bufs[s.buf[0]], bufs[s.buf[1]], bufs[s.buf[2]],
               bufs[s.buf[3]], bufs[s.buf[4]], s.n[0], s.n[1], s.n[2], s.n[3], s.n[4], s.off[0], s.off[2], s.n[5], s.n[6], s.f[0], s.f[1], (uint32_t)n_sm);
}

// ── CAUSAL_CONV ──────────────────────────────────────────────────────────────────────────────────────────────────
template <typename WT>
__global__ void k_causal_conv(float* __restrict__ dst, const float* __restrict__ src, const WT* __restrict__ w, float* state,
                              const float* __restrict__ ctl, uint32_t T, uint32_t C, uint32_t taps, uint32_t src_rs, uint32_t dst_rs, uint32_t act,
                              uint32_t advance, const WT* __restrict__ bias) {
    pdl_enter();
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (size_t)T * C) return;
    const uint32_t t = (uint32_t)(e / C), c = (uint32_t)(e % C);
    float* st = state + (size_t)ctl_word(ctl, ZG_CTL_SLOT) * (taps - 1) * C;
    float y = bias ? wld(bias, c) : 0.0f;
    for (uint32_t j = 0; j < taps; j++) {
        const int tau = (int)t - (int)(taps - 1) + (int)j;     // time relative to the step's first token
        const float x = tau >= 0 ? src[(size_t)tau * src_rs + c] : st[(size_t)(tau + (int)(taps - 1)) * C + c];
        y = fmaf(wld(w, (size_t)c * taps + j), x, y);
        // single-token steps: this thread alone touches the channel's carried inputs, so it also shifts them (input j moves to
        // row j - 1, which was read one trip earlier)
        if (advance && j > 0) st[(size_t)(j - 1) * C + c] = x;
    }
    if (act == 1) y = y * sigmoidf_(y);
    dst[(size_t)t * dst_rs + c] = y;
}
// state row r holds the input of time (first token of the NEXT step) - (taps - 1) + r; rows ascend, so shifting in place is safe
__global__ void k_conv_advance(float* __restrict__ state, const float* __restrict__ src, const float* __restrict__ ctl, uint32_t T, uint32_t C,
                               uint32_t taps, uint32_t src_rs) {
    pdl_enter();
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) return;
    float* st = state + (size_t)ctl_word(ctl, ZG_CTL_SLOT) * (taps - 1) * C;
    for (uint32_t r = 0; r + 1 < taps; r++) {
        const int tau = (int)T - (int)(taps - 1) + (int)r;
        st[(size_t)r * C + c] = tau >= 0 ? src[(size_t)tau * src_rs + c] : st[(size_t)(r + T) * C + c];
    }
}

// ── DELTA_RULE ───────────────────────────────────────────────────────────────────────────────────────────────────
// Columns of the state evolve independently given the token's k, q, decay and beta, so a head is split by value columns
// over CTAs.  A thread keeps kDeltaRows consecutive key rows of one column in registers; the RS threads of a column sit in
// adjacent lanes and meet by shuffles.  The per-token vectors (unit k, scaled unit q, decay) of kDeltaTile tokens are
// prepared by the whole CTA at once, then the tokens are walked without further barriers.
constexpr int kDeltaRows = 16, kDeltaTile = 16, kDeltaThreads = 128;
// forms of the rule (op parameter n10): plain accumulation without unit vectors and correction (gated linear attention), the
// decay as a tempered sigmoid, a SiLU output gate, an output scale, one decay per head instead of one per key channel
// a read-out before the token's write with the token itself joining through a bonus per key channel (RWKV's time mixing), the decay
// as exp(-exp(z)), an output norm whose weight is one vector over all heads
constexpr uint32_t kDeltaPlain = 1, kDeltaSigmoidDecay = 2, kDeltaSiluGate = 4, kDeltaOutScale = 8, kDeltaHeadDecay = 16, kDeltaBonus = 32, kDeltaExpDecay = 64, kDeltaWideNorm = 128;
// decay of one key channel from its logit z (the bias is already added): exp(-exp(A) softplus(z)), or sigmoid(z)^(1 / tau) =
// exp(-softplus(-z) / tau), or exp(-exp(z))
__device__ __forceinline__ float delta_decay(float z, float Ah, uint32_t form, float inv_tau) {
    if (form & kDeltaExpDecay) return expf(-expf(z));
    return (form & kDeltaSigmoidDecay) ? expf(-softplusf_(-z) * inv_tau) : expf(-Ah * softplusf_(z));
}
template <typename WT>
__global__ void __launch_bounds__(kDeltaThreads) k_delta_rule(
    float* __restrict__ dst, const float* __restrict__ qkv, const float* __restrict__ betab, const float* __restrict__ ab, const WT* __restrict__ wts,
    float* __restrict__ state, const float* __restrict__ ctl, uint32_t T, uint32_t H, uint32_t G, uint32_t dim, uint32_t vdim, uint32_t RS,
    uint32_t q_off, uint32_t k_off, uint32_t v_off, uint32_t beta_off, uint32_t A_off, uint32_t dt_off, uint32_t qkv_rs, uint32_t beta_rs,
    uint32_t a_rs, float unit_eps, float q_scale, uint32_t form, float inv_tau, uint32_t dst_rs, uint32_t u_off) {
    pdl_enter();
    extern __shared__ float sm[];
    const bool plain = form & kDeltaPlain;             // no unit vectors, no correction: S <- g S + k v^T
    const bool head_decay = form & kDeltaHeadDecay;    // a row of `ab` holds one logit per head
    const bool bonus = form & kDeltaBonus;             // plain: o = S^T q + (sum_i q_i u_i k_i) v before the write
    const uint32_t dpad = RS * kDeltaRows;             // rows incl. padding (k = q = 0, decay = 1 there)
    float* sk = sm;                                    // [tile][dpad]
    float* sq = sk + kDeltaTile * dpad;
    float* sg = sq + kDeltaTile * dpad;
    float* sbeta = sg + kDeltaTile * dpad;             // [tile]
    const uint32_t h = blockIdx.y, kv = h / (H / G);
    const uint32_t cols_per_cta = kDeltaThreads / RS;
    const uint32_t r = threadIdx.x % RS, col = blockIdx.x * cols_per_cta + threadIdx.x / RS;
    const bool live = col < vdim;
    const uint32_t slot = (uint32_t)ctl_word(ctl, ZG_CTL_SLOT);
    float* S_g = state + (((size_t)slot * H + h) * dim) * vdim;
    float S[kDeltaRows];
#pragma unroll
    for (int i = 0; i < kDeltaRows; i++) {
        const uint32_t row = r * kDeltaRows + i;
        S[i] = (live && row < dim) ? S_g[(size_t)row * vdim + col] : 0.0f;
    }
    const float Ah = (form & (kDeltaSigmoidDecay | kDeltaExpDecay)) ? 0.0f : expf(wld(wts, (size_t)A_off + h));
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (uint32_t t0 = 0; t0 < T; t0 += kDeltaTile) {
        const uint32_t nt = min((uint32_t)kDeltaTile, T - t0);
        __syncthreads();
        // prepare: warp w takes tokens w, w + 4, ...
        for (uint32_t tt = warp; tt < nt; tt += kDeltaThreads / 32) {
            const uint32_t t = t0 + tt;
            const float* qr = qkv + (size_t)t * qkv_rs + q_off + (size_t)kv * dim;
            const float* kr = qkv + (size_t)t * qkv_rs + k_off + (size_t)kv * dim;
            const float* ar = ab + (size_t)t * a_rs + (head_decay ? (size_t)h : (size_t)h * dim);
            const float gh = head_decay ? delta_decay(ar[0] + wld(wts, (size_t)dt_off + h), Ah, form, inv_tau) : 1.0f;
            float qn = q_scale, kn = 1.0f;
            if (!plain) {
                float qq = 0.0f, kk = 0.0f;
                for (uint32_t c = lane; c < dim; c += 32) { qq = fmaf(qr[c], qr[c], qq); kk = fmaf(kr[c], kr[c], kk); }
                qn = q_scale / sqrtf(warp_sum(qq) + unit_eps); kn = 1.0f / sqrtf(warp_sum(kk) + unit_eps);
            }
            for (uint32_t c = lane; c < dpad; c += 32) {
                const bool in = c < dim;
                sk[tt * dpad + c] = in ? kr[c] * kn : 0.0f;
                sq[tt * dpad + c] = in ? qr[c] * qn : 0.0f;
                sg[tt * dpad + c] = head_decay ? gh : in ? delta_decay(ar[c] + wld(wts, (size_t)dt_off + (size_t)h * dim + c), Ah, form, inv_tau) : 1.0f;
            }
            float own = 1.0f;
            if (bonus) {
                own = 0.0f;
                for (uint32_t c = lane; c < dim; c += 32) own = fmaf(qr[c] * qn * kr[c], wld(wts, (size_t)u_off + (size_t)h * dim + c), own);
                own = warp_sum(own);
            }
            if (lane == 0) sbeta[tt] = plain ? own : sigmoidf_(betab[(size_t)t * beta_rs + beta_off + h]);
        }
        float vt[kDeltaTile];                              // the tile's values of this column: independent loads, issued together
#pragma unroll
        for (int tt = 0; tt < kDeltaTile; tt++)
            vt[tt] = (live && (uint32_t)tt < nt) ? qkv[(size_t)(t0 + tt) * qkv_rs + v_off + (size_t)h * vdim + col] : 0.0f;
        __syncthreads();
#pragma unroll
        for (int tti = 0; tti < kDeltaTile; tti++) {
            const uint32_t tt = (uint32_t)tti;
            if (tt >= nt) break;
            const uint32_t t = t0 + tt;
            const float* k = sk + tt * dpad + r * kDeltaRows;
            const float* q = sq + tt * dpad + r * kDeltaRows;
            const float* g = sg + tt * dpad + r * kDeltaRows;
            const float v = vt[tti];
            if (bonus) {                                   // read first, then decay and write
                float os = 0.0f;
#pragma unroll
                for (int i = 0; i < kDeltaRows; i++) { os = fmaf(S[i], q[i], os); S[i] = fmaf(S[i], g[i], k[i] * v); }
                for (uint32_t o = 1; o < RS; o <<= 1) os += __shfl_xor_sync(0xffffffffu, os, o);
                if (live && r == 0) dst[(size_t)t * dst_rs + (size_t)h * vdim + col] = fmaf(sbeta[tt], v, os);
                continue;
            }
            float ks = 0.0f;
#pragma unroll
            for (int i = 0; i < kDeltaRows; i++) { S[i] *= g[i]; ks = fmaf(S[i], k[i], ks); }
            if (!plain) for (uint32_t o = 1; o < RS; o <<= 1) ks += __shfl_xor_sync(0xffffffffu, ks, o);
            const float u = plain ? v : sbeta[tt] * (v - ks);
            float os = 0.0f;
#pragma unroll
            for (int i = 0; i < kDeltaRows; i++) { S[i] = fmaf(k[i], u, S[i]); os = fmaf(S[i], q[i], os); }
            for (uint32_t o = 1; o < RS; o <<= 1) os += __shfl_xor_sync(0xffffffffu, os, o);
            if (live && r == 0) dst[(size_t)t * dst_rs + (size_t)h * vdim + col] = os;
        }
    }
#pragma unroll
    for (int i = 0; i < kDeltaRows; i++) {
        const uint32_t row = r * kDeltaRows + i;
        if (live && row < dim) S_g[(size_t)row * vdim + col] = S[i];
    }
}
// Prefill form of DELTA_RULE (kDeltaPrepMinTokens or more tokens, but for the short steps of delta_by_blocks): chunks of 16 tokens.  With D_l the decay of token l of a chunk (a diagonal) and S the
// state before it, every token's two products follow from products with S itself:
//   S_j^T x = S^T (D_1 .. D_j x) + sum_{i <= j} (x^T D_{i+1} .. D_j k_i) u_i,   u_j = beta_j (v_j - A_j^T S - sum_{i < j} ckk_ij u_i).
// Both are affine in S, so the triangular solve is done ahead, on the vectors instead of on the state's columns:
//   u_j = Vt_j - W_j^T S,   W_j = beta_j (A_j - sum_{i < j} ckk_ij W_i),   Vt_j = beta_j (v_j - sum_{i < j} ckk_ij Vt_i),
//   o_j = Vo_j + Q'_j^T S,  Q'_j = Q_j - sum_{i <= j} cqk_ij W_i,          Vo_j = sum_{i <= j} cqk_ij Vt_i,   S <- Gamma S + sum_j B_j u_j^T.
// k_delta_prepare does that for all chunks at once; what is left in sequence, k_delta_walk, is two small products per chunk.  Only products of decays
// occur (nothing is divided by one), so the form is as sound as token by token for any decay, and a token's row of any term depends on the tokens up to
// it alone.  A plain accumulation (u = v) has no W.
// Steps are walked in passes of at most kDeltaScratch bytes of prepared vectors: they stay in the L2 between the two kernels.
constexpr int kDeltaPrepMinTokens = 16;
constexpr uint32_t kWalkChunk = 16, kWalkMaxDim = 512, kWalkCols = 16;
constexpr size_t kDeltaScratch = 64u << 20;
// key rows a chunk's vectors are padded to: sixteen per warp and slice of the walk
__host__ __device__ constexpr uint32_t delta_rows(uint32_t dim) { return dim <= 64 ? 64 : dim <= 128 ? 128 : dim <= 256 ? 256 : 512; }
// a chunk's vectors as the walk stages them: [W | Q'] of dpad + 8 rows each (the lanes of a read lie in different banks), B as [row][16 tokens], Gamma ...
__host__ __device__ constexpr uint32_t delta_vec_elems(uint32_t dpad, bool plain) { return (plain ? 1 : 2) * kWalkChunk * (dpad + 8) + (kWalkChunk + 1) * dpad; }
// ... and with [Vt | Vo] of 16 tokens and 16 value columns at a time behind them, in the order of the accumulators that hold such a square
__host__ __device__ constexpr size_t delta_chunk_elems(uint32_t dpad, bool plain, uint32_t vdim) { return delta_vec_elems(dpad, plain) + (size_t)(vdim + kWalkCols - 1) / kWalkCols * 512; }
__host__ __device__ constexpr uint32_t delta_square(uint32_t tok, uint32_t col) { return (tok >> 3) * 128 + ((col & 7) * 4 + ((tok >> 1) & 3)) * 4 + (col >> 3) * 2 + (tok & 1); }
static uint32_t delta_pass_chunks(uint32_t T, uint32_t H, uint32_t dim, uint32_t vdim, bool plain) {
    const size_t one = delta_chunk_elems(delta_rows(dim), plain, vdim) * H * sizeof(float), most = kDeltaScratch / one;
    const uint32_t chunks = (T + kWalkChunk - 1) / kWalkChunk;
    return (uint32_t)(most < 4 ? chunks < 4 ? chunks : 4 : most < chunks ? most : chunks);
}
// One CTA per (chunk, head): units, scales and decays into shared memory; the 256 products between the tokens (136 q k, 120 k k), a warp for two of the
// tokens that wrote, four later tokens at a time; then a thread for a column of [A | V], whose solves are alike.  Loops are kept rolled where the data
// allows it: a straight line of 5000 instructions took 88 us where this takes 43 (1024 tokens, 16 heads of 128 x 128, launches alone): every CTA fetched it anew.
constexpr uint32_t kDeltaPrepThreads = 256;
constexpr uint32_t delta_prep_smem(uint32_t dpad) { return (3 * kWalkChunk + 2) * (dpad + 4) * 4; }
template <typename WT>
__global__ void __launch_bounds__(kDeltaPrepThreads, 2) k_delta_prepare(float* __restrict__ prep, const float* __restrict__ qkv, const float* __restrict__ betab, const float* __restrict__ ab,
                                const WT* __restrict__ wts, uint32_t T, uint32_t H, uint32_t G, uint32_t dim, uint32_t vdim, uint32_t dpad, uint32_t q_off,
                                uint32_t k_off, uint32_t v_off, uint32_t beta_off, uint32_t A_off, uint32_t dt_off, uint32_t qkv_rs, uint32_t beta_rs, uint32_t a_rs,
                                float unit_eps, float q_scale, uint32_t form, float inv_tau, uint32_t u_off, uint32_t early) {
    if (early) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    constexpr uint32_t C = kWalkChunk;
    const uint32_t NT = blockDim.x, warps = NT >> 5;                 // 4 or 8 warps
    extern __shared__ __align__(16) float sm[];
    __shared__ __align__(16) float qk[C][C], kk[C][C], scale[2 * C], beta[C];      // [j][i]
    const bool plain = form & kDeltaPlain, head_decay = form & kDeltaHeadDecay, bonus = form & kDeltaBonus;
    const uint32_t h = blockIdx.x, b = blockIdx.y, kv = h / (H / G), n = min(C, T - b * C), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, dp = dpad + 4;
    float* sk = sm;                                                  // [token][dp]
    float* sq = sk + C * dp;
    float* sd = sq + C * dp;
    float* sbias = sd + C * dp;
    float* sown = sbias + dp;
    const float* row0 = qkv + (size_t)b * C * qkv_rs;
    const float* ar = ab + (size_t)b * C * a_rs + (head_decay ? (size_t)h : (size_t)h * dim);
    for (uint32_t c = tid; c < dpad; c += NT) {
        sbias[c] = c < dim ? wld(wts, (size_t)dt_off + (head_decay ? (size_t)h : (size_t)h * dim + c)) : 0.0f;
        sown[c] = bonus && c < dim ? wld(wts, (size_t)u_off + (size_t)h * dim + c) : 1.0f;
    }
    const float Ah = (form & (kDeltaSigmoidDecay | kDeltaExpDecay)) ? 0.0f : expf(wld(wts, (size_t)A_off + h));
    if (tid < C) beta[tid] = plain || tid >= n ? 0.0f : sigmoidf_(betab[((size_t)b * C + tid) * beta_rs + beta_off + h]);
    // tokens past the step's end: nothing is written, nothing decays
    for (uint32_t j0 = warp; j0 < C; j0 += 2 * warps) {              // tokens j0 and j0 + warps
        float sums[4] = {};                                          // q q of the two, k k
        for (uint32_t c0 = 0; c0 < dpad; c0 += 128) {
            float x[2][3][4];
#pragma unroll
            for (int l = 0; l < 2; l++)
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const uint32_t c = c0 + lane + 32 * i, j = j0 + l * warps;
                    const bool on = c < dim && j < n;
                    const float* r = row0 + (size_t)j * qkv_rs + (size_t)kv * dim + c;
                    x[l][0][i] = on ? r[q_off] : 0.0f;
                    x[l][1][i] = on ? r[k_off] : 0.0f;
                    x[l][2][i] = on ? ar[(size_t)j * a_rs + (head_decay ? 0 : c)] : 0.0f;
                }
#pragma unroll
            for (int l = 0; l < 2; l++)
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const uint32_t c = c0 + lane + 32 * i, at = (j0 + l * warps) * dp + c;
                    sums[l] = fmaf(x[l][0][i], x[l][0][i], sums[l]);
                    sums[2 + l] = fmaf(x[l][1][i], x[l][1][i], sums[2 + l]);
                    if (c < dpad) { sq[at] = x[l][0][i]; sk[at] = x[l][1][i]; sd[at] = x[l][2][i]; }
                }
        }
        const float total = reduce_scatter<4>(sums, lane);           // lane l: q of token j0 + l warps, lane 2 + l: k
        if (lane < 4) {
            const float own = lane < 2 ? q_scale : 1.0f;
            scale[(lane & 2) * 8 + j0 + (lane & 1) * warps] = plain ? own : own / sqrtf(total + unit_eps);
        }
    }
    __syncthreads();
    const uint32_t width = min(dpad, NT), at_once = NT / width;      // fewer rows than threads: several tokens at a time
    for (uint32_t c = tid & (width - 1); c < dpad; c += width) {
        const float bias = sbias[c];
#pragma unroll 2
        for (uint32_t j = tid / width; j < C; j += at_once) {
            const uint32_t at = j * dp + c;
            sq[at] *= scale[j];
            sk[at] *= scale[C + j];
            sd[at] = c < dim && j < n ? delta_decay(sd[at] + bias, Ah, form, inv_tau) : 1.0f;
        }
    }
    __syncthreads();
    auto dot = [](float4 a, float4 b) { return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, a.w * b.w))); };
#pragma unroll 1
    for (uint32_t m = 2 * warp; m < C; m += m & 1 ? 2 * warps - 1 : 1) {      // tokens m / 2 and 15 - m / 2 have 17 later ones and themselves together
        const uint32_t i = m & 1 ? C - 1 - (m >> 1) : m >> 1;
#pragma unroll 1
        for (uint32_t c0 = 4 * lane; c0 < max(dpad, 128u); c0 += 128) {
            const bool on = c0 < dpad;
            const uint32_t c = on ? c0 : 0;                          // 64 rows: the upper lanes hold zeros
            float4 d = *reinterpret_cast<const float4*>(sk + i * dp + c);      // what token i wrote, as the later tokens find it
            if (!on) d = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const float4 own = *reinterpret_cast<const float4*>(sown + c), q = *reinterpret_cast<const float4*>(sq + i * dp + c);
            const float self = warp_sum(dot(make_float4(q.x * own.x, q.y * own.y, q.z * own.z, q.w * own.w), d));
            if (lane == 0) qk[i][i] = c0 < 128 ? self : qk[i][i] + self;
#pragma unroll 1
            for (uint32_t j0 = i + 1; j0 < C; j0 += 4) {
                float v[8];                                          // q k of four tokens, k k of them
#pragma unroll
                for (int l = 0; l < 4; l++) {
                    const uint32_t at = min(j0 + l, C - 1) * dp + c;
                    const float4 g = *reinterpret_cast<const float4*>(sd + at), qj = *reinterpret_cast<const float4*>(sq + at), kj = *reinterpret_cast<const float4*>(sk + at);
                    if (bonus) v[l] = dot(qj, d);
                    d.x *= g.x; d.y *= g.y; d.z *= g.z; d.w *= g.w;
                    if (!bonus) v[l] = dot(qj, d);
                    v[4 + l] = dot(kj, d);
                }
                const float total = reduce_scatter<8>(v, lane);
                const uint32_t j = j0 + (lane & 3);
                if (lane < 8 && j < C) {
                    float& to = lane < 4 ? qk[j][i] : kk[j][i];
                    to = c0 < 128 ? total : to + total;
                }
            }
        }
    }
    __syncthreads();
    float* P = prep + ((size_t)h * gridDim.y + b) * delta_chunk_elems(dpad, plain, vdim);
    float* PQ = P + (plain ? 0 : C) * (dpad + 8);
    float* PB = P + (plain ? 1 : 2) * C * (dpad + 8);
    float* PV = P + delta_vec_elems(dpad, plain);
    const uint32_t vpad = (vdim + kWalkCols - 1) / kWalkCols * kWalkCols;
#pragma unroll 1
    for (uint32_t c = tid; c < dpad + vpad; c += NT) {
        const bool key = c < dpad;
        const uint32_t col = c - dpad;
        float y[C], z[C];                                            // key row: A then W, Q then Q'; value column: v then Vt, 0 then -Vo
        if (key) {
            float g = 1.0f, s = 1.0f, B[4];
#pragma unroll
            for (int j = 0; j < (int)C; j++) {
                const float before = g;
                g *= sd[j * dp + c];
                y[j] = sk[j * dp + c] * g;
                z[j] = sq[j * dp + c] * (bonus ? before : g);        // the bonus form reads the state before the token decays it
            }
            PB[(size_t)C * dpad + c] = g;
            // the upper and lower eight tokens change places in every other pair of rows (banks of the walk's reads)
            float* to = PB + (size_t)c * C;
            const uint32_t turn = ((c >> 1) & 1) << 3;
#pragma unroll
            for (int j = C - 1; j >= 0; j--) {
                B[j & 3] = s * sk[j * dp + c];
                s *= sd[j * dp + c];
                if ((j & 3) == 0) *reinterpret_cast<float4*>(to + ((uint32_t)j ^ turn)) = make_float4(B[0], B[1], B[2], B[3]);
            }
        } else {
            const float* vr = row0 + v_off + (size_t)h * vdim + col;
#pragma unroll
            for (int j = 0; j < (int)C; j++) { y[j] = col < vdim && (uint32_t)j < n ? vr[(size_t)j * qkv_rs] : 0.0f; z[j] = 0.0f; }
        }
        // what lies past the diagonal of a row is read but not used
#pragma unroll
        for (int j = 0; j < (int)C; j++) {
            if (!plain) {
#pragma unroll
                for (int i = 0; i < j; i += 4) {
                    const float4 r = *reinterpret_cast<const float4*>(&kk[j][i]);
                    const float c4[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
                    for (int l = 0; l < 4 && i + l < j; l++) y[j] = fmaf(-c4[l], y[i + l], y[j]);
                }
                y[j] *= beta[j];
            }
            if (!plain || !key) {
#pragma unroll
                for (int i = 0; i <= j; i += 4) {
                    const float4 r = *reinterpret_cast<const float4*>(&qk[j][i]);
                    const float c4[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
                    for (int l = 0; l < 4 && i + l <= j; l++) z[j] = fmaf(-c4[l], y[i + l], z[j]);
                }
            }
            asm volatile("" ::: "memory");                           // the coefficients of all rows at once would not fit the registers
        }
        if (key) {
#pragma unroll
            for (int j = 0; j < (int)C; j++) {
                if (!plain) P[(size_t)j * (dpad + 8) + c] = y[j];
                PQ[(size_t)j * (dpad + 8) + c] = z[j];
            }
        } else {
            float* to = PV + (size_t)(col / kWalkCols) * 512 + delta_square(0, col % kWalkCols);
#pragma unroll
            for (int j = 0; j < (int)C; j += 2) {
                *reinterpret_cast<float2*>(to + delta_square(j, 0)) = make_float2(y[j], y[j + 1]);
                *reinterpret_cast<float2*>(to + delta_square(j, 0) + 256) = make_float2(-z[j], -z[j + 1]);
            }
        }
    }
    if (!early) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");      // the walk's CTAs are placed when the GPU is theirs
}
__device__ __forceinline__ void mma_bf16_first(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {      // d = a b
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(0.0f));
}
// two pairs of values as an operand of three bfloat16 parts (24 bits)
__device__ __forceinline__ void split3_operand(const float* x, const float* y, uint32_t (&b)[3][2]) {
    const float2 u = *reinterpret_cast<const float2*>(x), v = *reinterpret_cast<const float2*>(y);
    split3(u.x, u.y, b[0][0], b[1][0], b[2][0]);
    split3(v.x, v.y, b[0][1], b[1][1], b[2][1]);
}
// acc[0] + acc[1] + acc[2] (first: =, else +=) a b: six products in chains of one, two and three
__device__ __forceinline__ void mma_split3(bool first, float (&acc)[3][4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][2]) {
    if (first) { mma_bf16_first(acc[2], a[2], b[0]); mma_bf16_first(acc[1], a[1], b[0]); mma_bf16_first(acc[0], a[0], b[0]); }
    else { mma_bf16(acc[2], a[2], b[0]); mma_bf16(acc[1], a[1], b[0]); mma_bf16(acc[0], a[0], b[0]); }
    mma_bf16(acc[2], a[0], b[2]);
    mma_bf16(acc[1], a[0], b[1]);
    mma_bf16(acc[2], a[1], b[1]);
}
// A CTA owns 16 value columns of a head.  WARPS warps hold SL slices of 16 key rows of S^T each, in registers, as f32 accumulators of mma.sync: the same
// registers, split into three bfloat16 parts, are the A operand of the next chunk's products.  Per chunk they form their shares of W S, sum those over
// the warps, and update S <- Gamma S + B u; as many warps beside them read the parts of S from shared memory and form the outputs Q' S + Vo, off the chain from
// chunk to chunk.  The products are far too small for tcgen05 (16 x 32 x 128 and 128 x 16 x 16, each waiting for the one before).  Measured at 1024
// tokens, 16 heads of 128 x 128: 75 us; with the outputs formed by the warps that hold S 84 us, with f32 FMAs 128 us (bound by what shared memory
// delivers to registers, 128 bytes a clock: 2500 clocks a chunk), four tokens at a time on one solve each 176 us.
constexpr uint32_t kWalkStages = 3, kWalkAlone = 116 * 1024;      // the latter: bytes of shared memory of a CTA that is to have an SM to itself
constexpr uint32_t delta_walk_smem(uint32_t dpad, bool plain, uint32_t warps, uint32_t stages) {
    return (stages * (delta_vec_elems(dpad, plain) + 512) + 2 * dpad / 16 * 384 + warps * 512) * 4 + 3 * 256 * 2 + 8 * kWalkStages;
}
// Columns of a CTA's 16 (`which`) as plain f32 sums, by all of its threads: where the state, a vector or a u rounds to infinity as bfloat16 or is not finite, its parts are no
// numbers though the sums may be.  Outputs that are finite stay.  sm: dpad + 16 rows of 16; dst, S_g: at the first column.
template <uint32_t dpad, bool PLAIN>
__device__ __forceinline__ void delta_walk_plain(float* sm, const float* P, size_t stride, float* dst, uint32_t dst_rs, float* S_g, uint32_t T, uint32_t dim, uint32_t vdim, uint32_t cols,
                                              uint32_t which) {
    constexpr uint32_t C = kWalkChunk, QR = PLAIN ? 0 : C, xs = dpad + 8, vec_elems = delta_vec_elems(dpad, PLAIN);
    float* S = sm;                                                    // [row][16]
    float* u = sm + dpad * kWalkCols;                                 // [token][16]
    const uint32_t col = threadIdx.x % kWalkCols, first = threadIdx.x / kWalkCols, step = blockDim.x / kWalkCols;
    const bool on = col < cols && (which >> col & 1);
    for (uint32_t row = first; row < dim; row += step) S[row * kWalkCols + col] = on ? S_g[(size_t)row * vdim + col] : 0.0f;
    __syncthreads();
#pragma unroll 1
    for (uint32_t t = 0; t < T; t += C, P += stride) {
        const float* B = P + (QR + C) * xs;
        const uint32_t n = min(C, T - t);
        for (uint32_t j = first; j < n; j += step) {
            const float* V = P + vec_elems + blockIdx.x * 512 + delta_square(j, col);
            float ws = 0.0f, qs = 0.0f;
            for (uint32_t row = 0; row < dim; row++) {
                const float x = S[row * kWalkCols + col];
                if (!PLAIN) ws = fmaf(P[j * xs + row], x, ws);
                qs = fmaf(P[(QR + j) * xs + row], x, qs);
            }
            u[j * kWalkCols + col] = V[0] - ws;
            float* o = dst + (size_t)(t + j) * dst_rs + col;
            if (on && !(fabsf(*o) <= 3.4028234e38f)) *o = V[256] + qs;
        }
        __syncthreads();
        for (uint32_t row = first; row < dim; row += step) {
            const uint32_t turn = ((row >> 1) & 1) << 3;
            float x = S[row * kWalkCols + col] * B[C * dpad + row];
            for (uint32_t j = 0; j < n; j++) x = fmaf(B[row * C + (j ^ turn)], u[j * kWalkCols + col], x);
            S[row * kWalkCols + col] = x;
        }
        __syncthreads();
    }
    if (on) for (uint32_t row = first; row < dim; row += step) S_g[(size_t)row * vdim + col] = S[row * kWalkCols + col];
}
// as a call: inlined into the kernels of 256 and 512 rows, it costs them registers (512 rows, 1024 tokens: 304 us, inlined 320)
template <uint32_t dpad, bool PLAIN>
__device__ __noinline__ void delta_walk_plain_call(float* sm, const float* P, size_t stride, float* dst, uint32_t dst_rs, float* S_g, uint32_t T, uint32_t dim, uint32_t vdim, uint32_t cols,
                                                   uint32_t which) {
    delta_walk_plain<dpad, PLAIN>(sm, P, stride, dst, dst_rs, S_g, T, dim, vdim, cols, which);
}
// (the second bound: 256 rows, 8 heads, 1024 tokens 151 us with it and 157 without; the others are left to the compiler)
template <int SL, int WARPS, bool PLAIN>
__global__ void __launch_bounds__(64 * WARPS, SL == 2 ? 1 : 0) k_delta_walk(float* __restrict__ dst, const float* __restrict__ prep, float* __restrict__ state, const float* __restrict__ ctl,
                                                           uint32_t T, uint32_t H, uint32_t dim, uint32_t vdim, uint32_t dst_rs, uint32_t stages) {
    extern __shared__ __align__(16) float sm[];
    __shared__ uint32_t failed, spoiled;                              // some thread's wait gave up: the CTA's outputs and its part of the state are not numbers; columns that are not finite
    constexpr uint32_t C = kWalkChunk, QR = PLAIN ? 0 : C, dpad = 16 * SL * WARPS, xs = dpad + 8, vec_elems = delta_vec_elems(dpad, PLAIN), NT = 32 * WARPS, PER = 256 / NT;
    constexpr uint32_t stage_elems = vec_elems + 512, slices = SL * WARPS;      // of a stage: the chunk's vectors, [Vt | Vo] of the CTA's columns
    const uint32_t h = blockIdx.y, col0 = blockIdx.x * kWalkCols, chunks = (T + C - 1) / C, tid = threadIdx.x % NT, lane = tid & 31, warp = tid >> 5;
    const bool outputs = threadIdx.x >= NT;                           // a warp's role
    float* parts = sm + stages * stage_elems;                         // parts of S^T: [chunk parity][slice][part][lane][4]
    float* part_u = parts + 2 * slices * 384;                         // [warp][256]
    float* part_o = part_u + WARPS * 256;                             // [warp][256]
    bf16* U = reinterpret_cast<bf16*>(part_o + WARPS * 256);          // [part][256]
    const uint32_t bars = smem_u32(U + 3 * 256);
    const size_t stride = delta_chunk_elems(dpad, PLAIN, vdim);
    const float* P = prep + (size_t)h * chunks * stride;
    if (threadIdx.x == NT) {
        failed = spoiled = 0;
        for (uint32_t i = 0; i < stages; i++) mbar_init(bars + 8 * i, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    auto state_of = [&] { return state + (((size_t)(uint32_t)ctl_word(ctl, ZG_CTL_SLOT) * H + h) * dim) * vdim + col0; };
    auto redo = [&] {                                                 // both roles, at the end: every copy has arrived, and of these columns the state in memory is that before the step
        auto plain = SL == 1 ? delta_walk_plain<dpad, PLAIN> : delta_walk_plain_call<dpad, PLAIN>;
        plain(sm, prep + (size_t)h * chunks * stride, stride, dst + (size_t)h * vdim + col0, dst_rs, state_of(), T, dim, vdim, vdim - col0, spoiled);
    };
    auto stage = [&](uint32_t b, uint32_t i) {                        // one thread; nobody reads stage i any more
        if (b >= chunks) return;
        const float* src = P + (size_t)b * stride;
        float* to = sm + i * stage_elems;
        mbar_expect_tx(bars + 8 * i, stage_elems * 4);
        bulk_load(to, src, vec_elems * 4, bars + 8 * i);
        bulk_load(to + vec_elems, src + vec_elems + blockIdx.x * 512, 2048, bars + 8 * i);
    };
    if (threadIdx.x == NT) for (uint32_t b = 0; b + 1 < stages || b == 0; b++) stage(b, b);
    const uint32_t g = lane >> 2, t = lane & 3;
    // element e of a chunk's 16 x 16 u or o, in the order of the accumulators that hold them
    auto tok_of = [](uint32_t e) { return (e >> 7) * 8 + 2 * ((e >> 2) & 3) + (e & 1); };
    auto col_of = [](uint32_t e) { return ((e >> 4) & 7) + 8 * ((e >> 1) & 1); };
    auto products = [&](const uint32_t (&b)[SL][2][3][2], auto part_of, float* out) {      // of 16 vectors with this warp's rows
        float acc[2][3][4];
#pragma unroll
        for (int s = 0; s < SL; s++) {
            uint32_t a[3][4];
            part_of(s, a);
#pragma unroll
            for (int i = 0; i < 2; i++) mma_split3(s == 0, acc[i], a, b[s][i]);
        }
#pragma unroll
        for (int i = 0; i < 2; i++) {
            float x[4];
#pragma unroll
            for (int r = 0; r < 4; r++) x[r] = acc[i][0][r] + (acc[i][1][r] + acc[i][2][r]);
            *reinterpret_cast<float4*>(out + i * 128 + lane * 4) = make_float4(x[0], x[1], x[2], x[3]);
        }
    };
    auto vectors = [&](const float* X, uint32_t (&b)[SL][2][3][2]) {
#pragma unroll
        for (int s = 0; s < SL; s++)
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const float* x = X + (8 * i + g) * xs + (s * WARPS + warp) * 16 + 2 * t;
                split3_operand(x, x + 8, b[s][i]);
            }
    };
    auto total = [&](const float* part) {                             // over the warps
        float x[4] = {};
#pragma unroll
        for (uint32_t w = 0; w < WARPS; w++) x[w & 3] += part[w * 256];
        return (x[0] + x[1]) + (x[2] + x[3]);
    };
    __syncthreads();                                                  // the barriers are there
    uint32_t cur = 0, parity = 0;
    auto turn_stage = [&](uint32_t b) {
        if (stages == 1) {                                            // no room for the next chunk's vectors beside this one's
            __syncthreads();
            if (threadIdx.x == NT) stage(b + 1, 0);
        }
        if (++cur == stages) { cur = 0; parity ^= 1; }
    };
    if (outputs) {
        float* to[PER];
        float zero[PER] = {};                                         // not zero once an output was not finite
#pragma unroll
        for (uint32_t p = 0; p < PER; p++) to[p] = dst + (size_t)tok_of(tid + p * NT) * dst_rs + (size_t)h * vdim + col0 + col_of(tid + p * NT);
        const size_t chunk_rs = (size_t)C * dst_rs;
#pragma unroll 1
        for (uint32_t b = 0; b < chunks; b++) {
            const float* X = sm + cur * stage_elems;
            if (!mbar_wait(bars + 8 * cur, parity)) failed = 1;
            uint32_t q[SL][2][3][2];
            vectors(X + QR * xs, q);
            __syncthreads();                                          // the parts of S are there, and the chunk before is done with
            if (stages > 1 && tid == 0) stage(b + stages - 1, cur == 0 ? stages - 1 : cur - 1);
            products(q, [&](int s, uint32_t (&a)[3][4]) {
#pragma unroll
                for (int i = 0; i < 3; i++) {
                    const uint4 x = *reinterpret_cast<const uint4*>(parts + (((b & 1) * slices + s * WARPS + warp) * 3 + i) * 128 + lane * 4);
                    a[i][0] = x.x; a[i][1] = x.y; a[i][2] = x.z; a[i][3] = x.w;
                }
            }, part_o + warp * 256);
            bar_sync(2, NT);
#pragma unroll
            for (uint32_t p = 0; p < PER; p++) {
                const uint32_t e = tid + p * NT;
                const float o = X[vec_elems + 256 + e] + total(part_o + e);
                zero[p] = fmaf(o, 0.0f, zero[p]);
                if (b * C + tok_of(e) < T && col0 + col_of(e) < vdim) *to[p] = o;
                to[p] += chunk_rs;
            }
            turn_stage(b);
        }
#pragma unroll
        for (uint32_t p = 0; p < PER; p++)
            if (zero[p] != 0.0f) atomicOr(&spoiled, 1u << col_of(tid + p * NT));
        __syncthreads();
        if (failed) {
            if (tid == 0) count_timeout();
            for (uint32_t e = tid; e < T * kWalkCols; e += NT)
                if (col0 + e % kWalkCols < vdim) dst[(size_t)(e / kWalkCols) * dst_rs + (size_t)h * vdim + col0 + e % kWalkCols] = __uint_as_float(0x7fffffffu);
        } else if (spoiled) redo();
        return;
    }
    // accumulator r of tile i of slice s: column g + 8 (r / 2), row 8 i + 2 t + r % 2 of the slice
    float* S_g = state_of();
    float S[SL][2][4];
    auto each_state = [&](auto f) {
#pragma unroll
        for (int s = 0; s < SL; s++)
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const uint32_t row = (s * WARPS + warp) * 16 + 8 * i + 2 * t + (r & 1), col = g + 8 * (r >> 1);
                    f(S[s][i][r], row < dim && col0 + col < vdim, (size_t)row * vdim + col, r >> 1);
                }
    };
    each_state([&](float& x, bool on, size_t at, int) { x = on ? S_g[at] : 0.0f; });
#pragma unroll 1
    for (uint32_t b = 0; b < chunks; b++) {
        const float* X = sm + cur * stage_elems;
        const float* B = X + (QR + C) * xs;
        uint32_t A[SL][3][4];
#pragma unroll
        for (int s = 0; s < SL; s++) {
#pragma unroll
            for (int i = 0; i < 4; i++) split3(S[s][i >> 1][2 * (i & 1)], S[s][i >> 1][2 * (i & 1) + 1], A[s][0][i], A[s][1][i], A[s][2][i]);
#pragma unroll
            for (int i = 0; i < 3; i++)
                *reinterpret_cast<uint4*>(parts + (((b & 1) * slices + s * WARPS + warp) * 3 + i) * 128 + lane * 4) = make_uint4(A[s][i][0], A[s][i][1], A[s][i][2], A[s][i][3]);
        }
        if (!mbar_wait(bars + 8 * cur, parity)) failed = 1;
        if (!PLAIN) {
            uint32_t w[SL][2][3][2];
            vectors(X, w);
            products(w, [&](int s, uint32_t (&a)[3][4]) {
#pragma unroll
                for (int i = 0; i < 12; i++) a[i >> 2][i & 3] = A[s][i >> 2][i & 3];
            }, part_u + warp * 256);
        }
        __syncthreads();                                              // the shares of u are there
#pragma unroll
        for (uint32_t p = 0; p < PER; p++) {
            const uint32_t e = tid + p * NT;
            float u = X[vec_elems + e];
            if (!PLAIN) u -= total(part_u + e);
#pragma unroll
            for (int i = 0; i < 3; i++) {
                const bf16 part = __float2bfloat16_rn(u);
                U[i * 256 + e] = part;
                u -= __bfloat162float(part);
            }
        }
        uint32_t rows[SL][2][3][2];
        float2 decay[SL][2];
#pragma unroll
        for (int s = 0; s < SL; s++)
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const uint32_t row0 = (s * WARPS + warp) * 16 + 8 * i, turn = ((g >> 1) & 1) << 3;
                const float* row = B + (row0 + g) * C;
                split3_operand(row + ((2 * t) ^ turn), row + ((2 * t + 8) ^ turn), rows[s][i]);
                decay[s][i] = *reinterpret_cast<const float2*>(B + C * dpad + row0 + 2 * t);
            }
        bar_sync(1, NT);                                              // u
        uint32_t UA[3][4];
#pragma unroll
        for (int i = 0; i < 3; i++) {
            const uint2 lo = *reinterpret_cast<const uint2*>(U + i * 256 + lane * 4), hi = *reinterpret_cast<const uint2*>(U + i * 256 + 128 + lane * 4);
            UA[i][0] = lo.x; UA[i][1] = lo.y; UA[i][2] = hi.x; UA[i][3] = hi.y;
        }
#pragma unroll
        for (int s = 0; s < SL; s++)
#pragma unroll
            for (int i = 0; i < 2; i++) {
                float acc[3][4];
                mma_split3(true, acc, UA, rows[s][i]);
#pragma unroll
                for (int r = 0; r < 4; r++) S[s][i][r] = fmaf(S[s][i][r], r & 1 ? decay[s][i].y : decay[s][i].x, acc[0][r] + (acc[1][r] + acc[2][r]));
            }
        turn_stage(b);
    }
    // (what is not finite on the way stays so in the state)
    float zero[2] = {};
    each_state([&](float& x, bool, size_t, int half) { zero[half] = fmaf(x, 0.0f, zero[half]); });
    if (zero[0] != 0.0f) atomicOr(&spoiled, 1u << g);
    if (zero[1] != 0.0f) atomicOr(&spoiled, 1u << (g + 8));
    __syncthreads();
    const bool ok = !failed;
    const uint32_t keep = ok ? ~spoiled : ~0u;
    each_state([&](float& x, bool on, size_t at, int half) {
        if (on && (keep >> (g + 8 * half) & 1)) S_g[at] = ok ? x : __uint_as_float(0x7fffffffu);
    });
    if (ok && spoiled) redo();
}
// Short prefill steps (delta_by_blocks): four tokens at a time, the triangular solve of four scalars per value column in the walk itself.  Preparing is cheap
// then (a warp per block of four tokens and head leaves [A_1 .. A_4 | Q_1 .. Q_4 | B_1 .. B_4 | Gamma] and the scalars [beta (4) | ckk (4 x 4) | cqk (4 x 4)], zero
// where i does not precede j, laid out [head][block]), but a block waits for the one before.  k_delta_block_walk streams the vectors into shared memory with cp.async,
// double buffered; a warp owns two value columns, a lane R key rows of both, and the 16 sums of a block (8 products, 2 columns) are reduced over the lanes by
// halving what is left each time: they end one per lane (column, k or q, token).
constexpr int kBlockThreads = 256, kBlockTokens = 4, kBlockScalars = 36, kBlockCols = 2;
__host__ __device__ constexpr uint32_t delta_block_elems(uint32_t dpad, bool plain) { return ((plain ? 2 : 3) * kBlockTokens + 1) * dpad + kBlockScalars; }
static uint32_t delta_block_rows(uint32_t dim) { return dim <= 64 ? 2 : 4; }      // key rows per lane
// Where that is faster than chunks of 16, whose fixed costs are larger.  Up to 64 key rows: below 32 tokens (2 heads of 64 x 64, 16 tokens: 10.1 us against 11.5,
// 24 tokens 11.7 against 12.4, 32 tokens 12.7 against 12.4), below 40 up to 32 rows (8 heads of 32 x 32: 32 tokens 11.2 against 12.0, 40 tokens equal), and up to 52 where the
// chunks' three launches have more CTAs than SMs and no longer start side by side (16 heads of 64 x 64, 24 tokens: 11.8 against 14.8, 52 tokens equal; 64 heads, 48 tokens
// 19.7 against 21.9; up to 40 where walk CTAs share SMs and their launch is early, or are more than two an SM: 40 heads, 48 tokens 19.5 against 17.7; 128 heads, 40 tokens
// 27.8 against 28.5, 48 tokens 32.4 against 29.6).  Up to 128 key rows only up to 24 tokens
// and where the chunks' walk has nearly an SM per CTA, so that the blocks' kernels do not start side by side either (16 heads of 128 x 128, 16 tokens: 15.4 against
// 16.5, 28 tokens equal; 10 heads 17.9 against 13.8; 24 heads 18.7 against 15.1).
constexpr uint32_t kBlockSideBySide = 100;             // CTAs of both kernels up to which the second is placed beside the first
static uint32_t delta_block_prep_ctas(uint32_t T, uint32_t H) { return ((T + kBlockTokens - 1) / kBlockTokens * H + 3) / 4; }
static bool delta_by_blocks(uint32_t T, uint32_t H, uint32_t dim, uint32_t vdim) {
    const uint32_t sms = zg_sm_count(), walk = (vdim + kWalkCols - 1) / kWalkCols * H;
    if (T > 52 || dim > 128) return false;
    if (dim > 64) return T <= 24 && walk <= sms && walk + delta_block_prep_ctas(T, H) > kBlockSideBySide;
    if (T < (dim <= 32 ? 40u : 32u)) return true;
    const uint32_t prep = (T + kWalkChunk - 1) / kWalkChunk * H;
    return prep + walk + (T * H + 3) / 4 > sms && (T <= 40 || walk <= sms || (prep > sms && walk <= 2 * sms));
}
template <typename WT, int R>
__global__ void k_delta_block_prepare(float* __restrict__ prep, const float* __restrict__ qkv, const float* __restrict__ betab, const float* __restrict__ ab,
                                const WT* __restrict__ wts, uint32_t T, uint32_t H, uint32_t G, uint32_t dim, uint32_t q_off,
                                uint32_t k_off, uint32_t beta_off, uint32_t A_off, uint32_t dt_off, uint32_t qkv_rs, uint32_t beta_rs, uint32_t a_rs,
                                float unit_eps, float q_scale, uint32_t form, float inv_tau, uint32_t u_off) {
    pdl_enter();
    constexpr int B = kBlockTokens;
    constexpr uint32_t dpad = 32 * R;
    const bool plain = form & kDeltaPlain, head_decay = form & kDeltaHeadDecay, bonus = form & kDeltaBonus;
    const uint32_t w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31, blocks = (T + B - 1) / B;
    if (w >= blocks * H) return;
    const uint32_t b = w / H, h = w % H, kv = h / (H / G), n = min((uint32_t)B, T - b * B);
    const float* qr = qkv + (size_t)b * B * qkv_rs + q_off + (size_t)kv * dim;
    const float* kr = qkv + (size_t)b * B * qkv_rs + k_off + (size_t)kv * dim;
    const float* ar = ab + (size_t)b * B * a_rs + (head_decay ? (size_t)h : (size_t)h * dim);
    float k[B][R], q[B][R], D[B][R];                                 // every load in flight at once
#pragma unroll
    for (int j = 0; j < B; j++)
#pragma unroll
        for (int i = 0; i < R; i++) {
            const uint32_t c = lane + 32 * i;
            const bool on = c < dim && (uint32_t)j < n;              // tokens past the step's end: nothing is written, nothing decays
            k[j][i] = on ? kr[(size_t)j * qkv_rs + c] : 0.0f;
            q[j][i] = on ? qr[(size_t)j * qkv_rs + c] : 0.0f;
            D[j][i] = on ? ar[(size_t)j * a_rs + (head_decay ? 0 : c)] : 0.0f;
        }
    float bias[R], own[R];
#pragma unroll
    for (int i = 0; i < R; i++) {
        const uint32_t c = lane + 32 * i;
        bias[i] = c < dim ? wld(wts, (size_t)dt_off + (head_decay ? (size_t)h : (size_t)h * dim + c)) : 0.0f;
        own[i] = bonus && c < dim ? wld(wts, (size_t)u_off + (size_t)h * dim + c) : 1.0f;
    }
    const float Ah = (form & (kDeltaSigmoidDecay | kDeltaExpDecay)) ? 0.0f : expf(wld(wts, (size_t)A_off + h));
    const float beta = plain || lane >= n ? 0.0f : betab[((size_t)b * B + lane) * beta_rs + beta_off + h];
    float scale = (lane & 4) ? 1.0f : q_scale;                       // lane j: of q_j, lane 4 + j: of k_j
    if (!plain) {
        float sq[2 * B];
#pragma unroll
        for (int j = 0; j < B; j++) {
            float qq = 0.0f, kk = 0.0f;
#pragma unroll
            for (int i = 0; i < R; i++) { qq = fmaf(q[j][i], q[j][i], qq); kk = fmaf(k[j][i], k[j][i], kk); }
            sq[j] = qq; sq[B + j] = kk;
        }
        scale /= sqrtf(reduce_scatter<2 * B>(sq, lane) + unit_eps);
    }
#pragma unroll
    for (int j = 0; j < B; j++) {
        const float qn = __shfl_sync(0xffffffffu, scale, j), kn = __shfl_sync(0xffffffffu, scale, B + j);
#pragma unroll
        for (int i = 0; i < R; i++) {
            k[j][i] *= kn; q[j][i] *= qn;
            if (i && head_decay) D[j][i] = D[j][0];                  // one decay for all rows (what lies past `dim` is zero, whatever its decay)
            else D[j][i] = lane + 32 * i < dim && (uint32_t)j < n ? delta_decay(D[j][i] + bias[i], Ah, form, inv_tau) : 1.0f;
        }
    }
    float* P = prep + ((size_t)h * blocks + b) * delta_block_elems(dpad, plain);
    float* PQ = P + (plain ? 0 : B) * dpad;
    float* PB = PQ + B * dpad;
    float c[16] = {};                                                // cqk_ij at j (j + 1) / 2 + i, ckk_ij at 10 + j (j - 1) / 2 + i
#pragma unroll
    for (int e = 0; e < R; e++) {
        const uint32_t at = lane + 32 * e;
        float g = 1.0f;
#pragma unroll
        for (int j = 0; j < B; j++) {
            const float before = g;
            g *= D[j][e];
            if (!plain) P[j * dpad + at] = g * k[j][e];
            PQ[j * dpad + at] = (bonus ? before : g) * q[j][e];       // the bonus form reads the state before the token decays it
        }
        PB[B * dpad + at] = g;
        float s = 1.0f;
#pragma unroll
        for (int j = B - 1; j >= 0; j--) { PB[j * dpad + at] = s * k[j][e]; s *= D[j][e]; }
#pragma unroll
        for (int i = 0; i < B; i++) {
            float& self = c[i * (i + 1) / 2 + i];
            self = fmaf(q[i][e] * own[e], k[i][e], self);
            float d = k[i][e];                                       // what token i wrote, as the later tokens find it
#pragma unroll
            for (int j = i + 1; j < B; j++) {
                float& qk = c[j * (j + 1) / 2 + i];
                if (bonus) qk = fmaf(q[j][e], d, qk);
                d *= D[j][e];
                if (!bonus) qk = fmaf(q[j][e], d, qk);
                if (!plain) { float& kk = c[10 + j * (j - 1) / 2 + i]; kk = fmaf(k[j][e], d, kk); }
            }
        }
    }
    float* sc = PB + (B + 1) * dpad;
    if (lane < (uint32_t)B) sc[lane] = plain || lane >= n ? 0.0f : sigmoidf_(beta);
    const uint32_t cj = (lane >> 2) & 3, ci = lane & 3;               // lane 4 j + i: ckk_ij, lane 16 + 4 j + i: cqk_ij
    const float total = reduce_scatter<16>(c, lane);
    const float mine = __shfl_sync(0xffffffffu, total, lane < 16 ? 10 + cj * (cj - 1) / 2 + ci : cj * (cj + 1) / 2 + ci);
    sc[B + lane] = (lane < 16 ? ci < cj : ci <= cj) ? mine : 0.0f;
}
__device__ __forceinline__ void cp_async16(float* smem_dst, const float* gmem_src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem_dst)), "l"(gmem_src) : "memory");
}
template <int R, bool PLAIN>                       // key rows per lane: 2 or 4
__global__ void __launch_bounds__(kBlockThreads) k_delta_block_walk(float* __restrict__ dst, const float* __restrict__ qkv, const float* __restrict__ prep,
                                                               float* __restrict__ state, const float* __restrict__ ctl, uint32_t T, uint32_t H,
                                                               uint32_t dim, uint32_t vdim, uint32_t v_off, uint32_t qkv_rs, uint32_t dst_rs) {
    pdl_enter();
    extern __shared__ __align__(16) float sm[];
    constexpr int B = kBlockTokens, C = kBlockCols, Q = PLAIN ? 0 : B, W = Q + B;      // vectors before Q's and before B's
    constexpr uint32_t dpad = 32 * R, block_elems = delta_block_elems(dpad, PLAIN), tile_blocks = kDeltaTile / B, tile_elems = tile_blocks * block_elems;
    const uint32_t h = blockIdx.y, blocks = (T + B - 1) / B, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t col0 = (blockIdx.x * (kBlockThreads / 32) + warp) * C;                     // the warp's first column
    const uint32_t slot = (uint32_t)ctl_word(ctl, ZG_CTL_SLOT);
    float* S_g = state + (((size_t)slot * H + h) * dim) * vdim;
    auto row_of = [&](int i) { return lane * R + (uint32_t)i; };
    float2 S[C][R / 2];
#pragma unroll
    for (int i = 0; i < R; i++)
#pragma unroll
        for (int c = 0; c < C; c++) {
            const float x = row_of(i) < dim && col0 + c < vdim ? S_g[(size_t)row_of(i) * vdim + col0 + c] : 0.0f;
            if (i & 1) S[c][i / 2].y = x; else S[c][i / 2].x = x;
        }
    const float* P = prep + (size_t)h * blocks * block_elems;
    auto stage = [&](uint32_t b0, float* buf) {        // blocks [b0, min(b0 + tile, blocks)): one contiguous run
        const uint32_t n4 = min(tile_blocks, blocks - b0) * block_elems / 4;
        const float* src = P + (size_t)b0 * block_elems;
        for (uint32_t i = threadIdx.x; i < n4; i += kBlockThreads) cp_async16(buf + 4 * i, src + 4 * i);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    stage(0, sm);
    // lane (column, k or q, token), twice: its value of a block, its place in the outputs
    const uint32_t lc = (lane >> 3) & 1, lj = lane & 3;
    const bool live = col0 + lc < vdim;
    const float* vbase = qkv + (size_t)lj * qkv_rs + v_off + (size_t)h * vdim + col0 + lc;
    float vt[tile_blocks], vn[tile_blocks];
#pragma unroll
    for (int i = 0; i < (int)tile_blocks; i++) vt[i] = live && i * B + lj < T ? vbase[(size_t)i * B * qkv_rs] : 0.0f;
    // R / 2 pairs of a prepared vector
    auto vec = [&](const float* v, float2 (&x)[R / 2]) {
        if (R == 4) {
            const float4 y = *reinterpret_cast<const float4*>(v + lane * 4);
            x[0] = make_float2(y.x, y.y); x[R / 2 - 1] = make_float2(y.z, y.w);
        } else x[0] = *reinterpret_cast<const float2*>(v + lane * 2);
    };
    uint32_t cur = 0;
    for (uint32_t t0 = 0; t0 < T; t0 += kDeltaTile, cur ^= 1) {
        const bool more = t0 + kDeltaTile < T;
        if (more) stage((t0 + kDeltaTile) / B, sm + (cur ^ 1) * tile_elems);   // its last readers passed the barrier that ended the tile before
#pragma unroll
        for (int i = 0; i < (int)tile_blocks; i++) vn[i] = live && t0 + kDeltaTile + i * B + lj < T ? vbase[(size_t)(t0 + kDeltaTile + i * B) * qkv_rs] : 0.0f;
        if (more) asm volatile("cp.async.wait_group 1;" ::: "memory"); else asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        const float* tile = sm + cur * tile_elems;
#pragma unroll
        for (int bi = 0; bi < (int)tile_blocks; bi++) {
            const uint32_t tb = t0 + bi * B;
            if (bi && tb >= T) break;
            const float* row = tile + bi * block_elems;
            const float* sc = row + (W + B + 1) * dpad;
            float sums[W * C];                                        // [column][product]
#pragma unroll
            for (int d = 0; d < W; d++) {
                float2 x[R / 2], acc[C];
                vec(row + d * dpad, x);
#pragma unroll
                for (int c = 0; c < C; c++) acc[c] = __fmul2_rn(S[c][0], x[0]);
#pragma unroll
                for (int i = 1; i < R / 2; i++)
#pragma unroll
                    for (int c = 0; c < C; c++) acc[c] = __ffma2_rn(S[c][i], x[i], acc[c]);
#pragma unroll
                for (int c = 0; c < C; c++) sums[c * W + d] = acc[c].x + acc[c].y;
            }
            float total = reduce_scatter<W * C>(sums, lane);
            if (PLAIN) total = __shfl_sync(0xffffffffu, total, lc * B + lj);
            float u[B], uc[C][B];
#pragma unroll
            for (int j = 0; j < B; j++) u[j] = __shfl_sync(0xffffffffu, PLAIN ? vt[bi] : vt[bi] - total, (lane & 8) + j);
            if (!PLAIN) {
                const float4 beta = *reinterpret_cast<const float4*>(sc);
                const float4 c1 = *reinterpret_cast<const float4*>(sc + B + 4), c2 = *reinterpret_cast<const float4*>(sc + B + 8), c3 = *reinterpret_cast<const float4*>(sc + B + 12);
                u[0] *= beta.x;
                u[1] = fmaf(-c1.x, u[0], u[1]) * beta.y;
                u[2] = fmaf(-c2.y, u[1], fmaf(-c2.x, u[0], u[2])) * beta.z;
                u[3] = fmaf(-c3.z, u[2], fmaf(-c3.y, u[1], fmaf(-c3.x, u[0], u[3]))) * beta.w;
            }
#pragma unroll
            for (int j = 0; j < B; j++) {
                const float other = __shfl_xor_sync(0xffffffffu, u[j], 8);
                uc[0][j] = lc ? other : u[j];
                uc[1][j] = lc ? u[j] : other;
            }
            {
                float2 x[R / 2];
                vec(row + (W + B) * dpad, x);
#pragma unroll
                for (int i = 0; i < R / 2; i++)
#pragma unroll
                    for (int c = 0; c < C; c++) S[c][i] = __fmul2_rn(S[c][i], x[i]);
#pragma unroll
                for (int j = 0; j < B; j++) {
                    vec(row + (W + j) * dpad, x);
#pragma unroll
                    for (int i = 0; i < R / 2; i++)
#pragma unroll
                        for (int c = 0; c < C; c++) S[c][i] = __ffma2_rn(x[i], make_float2(uc[c][j], uc[c][j]), S[c][i]);
                }
            }
            const float4 cq = *reinterpret_cast<const float4*>(sc + B + 16 + 4 * lj);
            total = fmaf(cq.x, u[0], total);                          // a later token's u is left out, not multiplied by zero: it need not be finite
            if (lj >= 1) total = fmaf(cq.y, u[1], total);
            if (lj >= 2) total = fmaf(cq.z, u[2], total);
            if (lj == 3) total = fmaf(cq.w, u[3], total);
            if (live && (lane & 20) == 4 && tb + lj < T) dst[(size_t)(tb + lj) * dst_rs + (size_t)h * vdim + col0 + lc] = total;
        }
#pragma unroll
        for (int i = 0; i < (int)tile_blocks; i++) vt[i] = vn[i];
        __syncthreads();                                   // everyone is done with this buffer: the next iteration refills it
    }
#pragma unroll
    for (int i = 0; i < R; i++)
#pragma unroll
        for (int c = 0; c < C; c++)
            if (row_of(i) < dim && col0 + c < vdim) S_g[(size_t)row_of(i) * vdim + col0 + c] = i & 1 ? S[c][i / 2].y : S[c][i / 2].x;
}
// o / rms(o) * norm_w * sigmoid(gate) (or silu(gate)) * out_scale, one warp per (token, head), in place
template <typename WT>
__global__ void k_delta_out(float* __restrict__ dst, const float* __restrict__ gate, const WT* __restrict__ wts, uint32_t TH, uint32_t H,
                            uint32_t vdim, uint32_t gate_rs, uint32_t nw_off, float eps, uint32_t dst_rs, uint32_t silu_gate, float out_scale, uint32_t wide_norm) {
    pdl_enter();
    const uint32_t item = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (item >= TH) return;
    const uint32_t t = item / H, h = item % H;
    float* o = dst + (size_t)t * dst_rs + (size_t)h * vdim;
    const float* g = gate + (size_t)t * gate_rs + (size_t)h * vdim;
    float q = 0.0f;
    for (uint32_t c = lane; c < vdim; c += 32) q = fmaf(o[c], o[c], q);
    const float inv = out_scale / sqrtf(warp_sum(q) / (float)vdim + eps);
    for (uint32_t c = lane; c < vdim; c += 32) o[c] = o[c] * inv * wld(wts, (size_t)nw_off + (wide_norm ? (size_t)h * vdim : 0) + c) * (silu_gate ? g[c] * sigmoidf_(g[c]) : sigmoidf_(g[c]));
}

// ── ROUTE: one warp per token ────────────────────────────────────────────────────────────────────────────────────
template <typename WT>
__global__ void k_route(float* __restrict__ dst, const float* __restrict__ logits, const WT* __restrict__ corr, uint32_t T, uint32_t NE, uint32_t top,
                        uint32_t logits_rs, uint32_t mode, uint32_t groups, uint32_t keep, float weight_scale) {
    pdl_enter();
    extern __shared__ float sm[];                      // [warps][NE + groups] choice scores, group scores
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t t = blockIdx.x * (blockDim.x >> 5) + warp;
    if (t >= T) return;
    const float* z = logits + (size_t)t * logits_rs;
    float* ch = sm + warp * (NE + groups);
    float mx = -INFINITY, inv = 0.0f;
    if (mode == 0) {
        for (uint32_t e = lane; e < NE; e += 32) mx = fmaxf(mx, z[e]);
        mx = warp_max(mx);
        float sum = 0.0f;
        for (uint32_t e = lane; e < NE; e += 32) sum += expf(z[e] - mx);
        inv = 1.0f / warp_sum(sum);
        for (uint32_t e = lane; e < NE; e += 32) ch[e] = expf(z[e] - mx) * inv + wld(corr, e);
    } else if (mode == 1) {
        for (uint32_t e = lane; e < NE; e += 32) ch[e] = z[e] + wld(corr, e);   // biased logits choose AND weigh
    } else {
        for (uint32_t e = lane; e < NE; e += 32) ch[e] = sigmoidf_(z[e]) + wld(corr, e);
        if (groups > 1) {                              // only outputs of the `keep` best groups stay eligible
            float* gs = ch + NE;
            const uint32_t per = NE / groups;
            __syncwarp();
            for (uint32_t g = lane; g < groups; g += 32) {   // a group scores the sum of its two largest choice scores
                float a = -INFINITY, b = -INFINITY;
                for (uint32_t e = g * per; e < (g + 1) * per; e++) {
                    const float v = ch[e];
                    if (v > a) { b = a; a = v; } else if (v > b) b = v;
                }
                gs[g] = per > 1 ? a + b : a;
            }
            __syncwarp();
            uint32_t kept_mine = 0;                    // bit i: group lane + 32 i is kept (groups <= 1024)
            for (uint32_t c = 0; c < keep; c++) {
                float best = -INFINITY; uint32_t bi = 0xFFFFFFFFu;
                for (uint32_t g = lane; g < groups; g += 32) if (!((kept_mine >> (g / 32)) & 1u) && (gs[g] > best || bi == 0xFFFFFFFFu)) { best = gs[g]; bi = g; }
                for (int o = 16; o > 0; o >>= 1) {
                    const float ob = __shfl_xor_sync(0xffffffffu, best, o);
                    const uint32_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
                    if (oi != 0xFFFFFFFFu && (bi == 0xFFFFFFFFu || ob > best || (ob == best && oi < bi))) { best = ob; bi = oi; }
                }
                if (bi != 0xFFFFFFFFu && bi % 32 == lane) kept_mine |= 1u << (bi / 32);
            }
            for (uint32_t g = lane; g < groups; g += 32)
                if (!((kept_mine >> (g / 32)) & 1u))
                    for (uint32_t e = g * per; e < (g + 1) * per; e++) ch[e] = -INFINITY;
        }
    }
    __syncwarp();
    float first = 0.0f, chosen_sum = 0.0f;             // mode 1 (lane 0): the largest chosen logit and the sum of exp(z - first)
    for (uint32_t c = 0; c < top; c++) {
        float best = -INFINITY; uint32_t bi = 0xFFFFFFFFu;
        for (uint32_t e = lane; e < NE; e += 32) if (ch[e] > best) { best = ch[e]; bi = e; }
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, o);
            const uint32_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
        }
        if (lane == 0) {
            float* out = dst + ((size_t)t * top + c) * 2;
            reinterpret_cast<int*>(out)[0] = (int)bi;
            if (mode == 0) out[1] = bi < NE ? expf(z[bi] - mx) * inv : 0.0f;
            else if (mode == 2) { out[1] = bi < NE ? sigmoidf_(z[bi]) : 0.0f; chosen_sum += out[1]; }
            else if (mode == 3) out[1] = bi < NE ? sigmoidf_(z[bi]) * weight_scale : 0.0f;
            else {
                if (c == 0) first = best;
                out[1] = bi < NE ? expf(best - first) : 0.0f;
                chosen_sum += out[1];
            }
            if (bi < NE) ch[bi] = -INFINITY;
        }
        __syncwarp();
    }
    if ((mode == 1 || mode == 2) && lane == 0) {
        const float norm = 1.0f / (mode == 2 ? chosen_sum + 1e-20f : chosen_sum);
        for (uint32_t c = 0; c < top; c++) dst[((size_t)t * top + c) * 2 + 1] *= norm;
    }
}

// dot of one weight row with an f32 vector by a whole warp (every lane gets the sum); 16-byte weight loads when aligned,
// four of them in flight per lane (a row is streamed once, so what hides HBM latency is the number of independent loads)
template <typename WT>
__device__ __forceinline__ float fma_vec4(const float* wv, const float* __restrict__ x, float acc) {
    constexpr int V = WVec<WT>::n;
#pragma unroll
    for (int i = 0; i < V / 4; i++) {
        const float4 xv = *reinterpret_cast<const float4*>(x + 4 * i);
        acc = fmaf(xv.x, wv[4 * i], fmaf(xv.y, wv[4 * i + 1], fmaf(xv.z, wv[4 * i + 2], fmaf(xv.w, wv[4 * i + 3], acc))));
    }
    return acc;
}
template <typename WT>
__device__ __forceinline__ float warp_dot(const WT* __restrict__ w, const float* __restrict__ x, uint32_t K, uint32_t lane) {
    constexpr int V = WVec<WT>::n;
    float acc = 0.0f;
    if (K % V == 0 && (reinterpret_cast<size_t>(w) & 15) == 0 && (reinterpret_cast<size_t>(x) & 15) == 0) {
        float a1 = 0.0f, a2 = 0.0f, a3 = 0.0f;
        uint32_t k = lane * V;
        for (; k + 96 * V < K; k += 128 * V) {
            float w0[V], w1[V], w2[V], w3[V];
            wld_vec<WT>(w + k, w0); wld_vec<WT>(w + k + 32 * V, w1); wld_vec<WT>(w + k + 64 * V, w2); wld_vec<WT>(w + k + 96 * V, w3);
            acc = fma_vec4<WT>(w0, x + k, acc); a1 = fma_vec4<WT>(w1, x + k + 32 * V, a1);
            a2 = fma_vec4<WT>(w2, x + k + 64 * V, a2); a3 = fma_vec4<WT>(w3, x + k + 96 * V, a3);
        }
        for (; k < K; k += 32 * V) {
            float w0[V];
            wld_vec<WT>(w + k, w0);
            acc = fma_vec4<WT>(w0, x + k, acc);
        }
        acc = (acc + a1) + (a2 + a3);
    } else {
        for (uint32_t k = lane; k < K; k += 32) acc = fmaf(x[k], wld(w, k), acc);
    }
    return warp_sum(acc);
}
// two rows against the same vector, their loads interleaved (the gate and up rows of an expert)
template <typename WT>
__device__ __forceinline__ void warp_dot2(const WT* __restrict__ wa, const WT* __restrict__ wb, const float* __restrict__ x, uint32_t K, uint32_t lane,
                                          float& ra, float& rb) {
    constexpr int V = WVec<WT>::n;
    if (K % V == 0 && (reinterpret_cast<size_t>(wa) & 15) == 0 && (reinterpret_cast<size_t>(wb) & 15) == 0 && (reinterpret_cast<size_t>(x) & 15) == 0) {
        float a0 = 0.0f, a1 = 0.0f, b0 = 0.0f, b1 = 0.0f;
        uint32_t k = lane * V;
        for (; k + 32 * V < K; k += 64 * V) {
            float p0[V], p1[V], q0[V], q1[V];
            wld_vec<WT>(wa + k, p0); wld_vec<WT>(wb + k, q0); wld_vec<WT>(wa + k + 32 * V, p1); wld_vec<WT>(wb + k + 32 * V, q1);
            a0 = fma_vec4<WT>(p0, x + k, a0); b0 = fma_vec4<WT>(q0, x + k, b0);
            a1 = fma_vec4<WT>(p1, x + k + 32 * V, a1); b1 = fma_vec4<WT>(q1, x + k + 32 * V, b1);
        }
        for (; k < K; k += 32 * V) {
            float p0[V], q0[V];
            wld_vec<WT>(wa + k, p0); wld_vec<WT>(wb + k, q0);
            a0 = fma_vec4<WT>(p0, x + k, a0); b0 = fma_vec4<WT>(q0, x + k, b0);
        }
        ra = warp_sum(a0 + a1); rb = warp_sum(b0 + b1);
    } else {
        ra = warp_dot(wa, x, K, lane); rb = warp_dot(wb, x, K, lane);
    }
}

// ── MOE_FFN, token-wise form: every (token, choice) pair streams the rows of its expert (decode and short steps) ────────
template <typename WT>
__global__ void k_moe_up(float* __restrict__ y, const float* __restrict__ src, const float* __restrict__ route, const WT* __restrict__ wg,
                         const WT* __restrict__ wu, uint32_t D, uint32_t ff, uint32_t E, uint32_t top, float limit, float alpha, float uoff, uint32_t stage) {
    pdl_enter();
    const uint32_t pair = blockIdx.y;                  // token * top + choice
    const uint32_t f = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const uint32_t e = (uint32_t)reinterpret_cast<const int*>(route)[2 * (size_t)pair];
    if (e >= E) return;                                // identity experts have no weights (uniform over the CTA)
    extern __shared__ __align__(16) float xsh[];       // the token's input, staged once per CTA when it fits
    const float* x = src + (size_t)(pair / top) * D;
    if (stage) {
        for (uint32_t c = threadIdx.x; c < D; c += blockDim.x) xsh[c] = x[c];
        __syncthreads();
        x = xsh;
    }
    if (f >= ff) return;
    const size_t row = ((size_t)e * ff + f) * D;
    float g, u;
    warp_dot2(wg + row, wu + row, x, D, lane, g, u);
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
    if (lane == 0) y[(size_t)pair * ff + f] = g * sigmoidf_(alpha * g) * (u + uoff);
}
template <typename WT>
__global__ void k_moe_down(float* __restrict__ dst, const float* __restrict__ src, const float* __restrict__ y, const float* __restrict__ route,
                           const WT* __restrict__ wd, uint32_t D, uint32_t ff, uint32_t E, uint32_t top) {
    pdl_enter();
    const uint32_t t = blockIdx.y;
    const uint32_t d = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (d >= D) return;
    float acc = 0.0f;
    for (uint32_t c = 0; c < top; c++) {               // fixed order: the result does not depend on the launch shape
        const size_t pair = (size_t)t * top + c;
        const uint32_t e = (uint32_t)reinterpret_cast<const int*>(route)[2 * pair];
        const float w = route[2 * pair + 1];
        const float v = e < E ? warp_dot(wd + ((size_t)e * D + d) * ff, y + pair * ff, ff, lane) : src[(size_t)t * D + d];
        acc = fmaf(w, v, acc);
    }
    if (lane == 0) dst[(size_t)t * D + d] = acc;
}

// ── MOE_FFN, grouped form (prefill on bfloat16 sessions): the step's (token, choice) pairs are sorted by expert, the rows are gathered as bf16, and the
// experts' products run as tiles of ONE tensor-core matmul for gate, up and activation and one for down (dense_gemm.cu), so an expert's weights are read
// once per run of up to 256 rows instead of once per token ──
constexpr uint32_t kMoeMinRun = 64;
struct MoeLayout {          // offsets in f32 slots inside the op's scratch operand
    uint32_t R, experts;         // (token, choice) pairs; experts that can have any
    size_t seg, row_pair, pos_of_pair, xs, yb, z, total;
};
__host__ __device__ inline size_t up4(size_t n) { return (n + 3) & ~(size_t)3; }
MoeLayout moe_layout(uint32_t T, uint32_t D, uint32_t ff, uint32_t E, uint32_t top) {
    MoeLayout L;
    L.R = T * top;
    L.experts = E < L.R ? E : L.R;
    size_t o = 0;
    L.seg = o; o = up4(o + (size_t)(L.experts + L.R / kMoeMinRun) * (sizeof(ZgExpertSegment) / 4));
    L.row_pair = o; o = up4(o + L.R);
    L.pos_of_pair = o; o = up4(o + L.R);
    L.xs = o; o = up4(o + (size_t)L.R * D / 2);
    L.yb = o; o = up4(o + (size_t)L.R * ff / 2);
    L.z = o; o = up4(o + (size_t)L.R * D);
    L.total = o;
    return L;
}
// Rows of a run at most.  Long runs read the weights least often; where they leave the GPU without a tile of gate and up per SM, what counts is the time of a
// tile, and the runs are shorter (395 tokens, two of 4 experts of 368 x 392, 28 tiles: 41 us with runs of 256 rows, 27 with 64).  The down product takes the
// same runs: chosen by the fewer tiles of the two, 1024 tokens of 4 experts of 256 x 2048 took 55 us instead of 70, but 300 tokens of 8 of 512 x 2048 41 instead of 35.
// (A launch's choice: the layout has room for the shortest runs, whatever machine sizes the scratch.)
uint32_t moe_run(const MoeLayout& L, uint32_t ff, uint32_t n_sm) {
    uint32_t run = kExpertSegmentRows;
    while (run > kMoeMinRun && (ff + 127) / 128 * (L.experts + L.R / run) < n_sm) run /= 2;
    return run;
}
constexpr uint32_t kMoeMaxExperts = 1024;
__global__ void __launch_bounds__(1024) k_moe_sort(const float* __restrict__ route, ZgExpertSegment* __restrict__ seg, int* __restrict__ row_pair,
                                                   int* __restrict__ pos_of_pair, uint32_t pairs, uint32_t E, uint32_t segments, uint32_t run) {
    pdl_enter();
    __shared__ int cnt[kMoeMaxExperts], off[kMoeMaxExperts];
    for (uint32_t e = threadIdx.x; e < E; e += blockDim.x) cnt[e] = 0;
    for (uint32_t r = threadIdx.x; r < pairs; r += blockDim.x) row_pair[r] = -1;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < pairs; i += blockDim.x) {
        const uint32_t e = (uint32_t)reinterpret_cast<const int*>(route)[2 * (size_t)i];
        if (e < E) atomicAdd(&cnt[e], 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int o = 0;
        uint32_t n = 0;
        for (uint32_t e = 0; e < E; e++) {
            off[e] = o;
            const int c = cnt[e], runs = (c + (int)run - 1) / (int)run;
            const int rows = runs ? ((c + runs - 1) / runs + 15) / 16 * 16 : 0;      // equal shares, of whole multiples of 16
            for (int r = 0; r < c; r += rows) seg[n++] = ZgExpertSegment{(int)e, o + r, min(rows, c - r)};
            o += c;
            cnt[e] = 0;                                  // becomes the expert's fill cursor
        }
        for (; n < segments; n++) seg[n] = ZgExpertSegment{0, 0, 0};
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < pairs; i += blockDim.x) {
        const uint32_t e = (uint32_t)reinterpret_cast<const int*>(route)[2 * (size_t)i];
        int pos = -1;
        if (e < E) { pos = off[e] + atomicAdd(&cnt[e], 1); row_pair[pos] = (int)i; }
        pos_of_pair[i] = pos;                            // which row a pair landed in does not change its result
    }
}
__global__ void k_moe_gather(uint32_t* __restrict__ xs, const float* __restrict__ src, const int* __restrict__ row_pair, uint32_t D, uint32_t top) {
    pdl_enter();
    const uint32_t r = blockIdx.x;
    const int pair = row_pair[r];
    if (pair < 0) return;                                // rows that no expert takes
    const float* x = src + (size_t)((uint32_t)pair / top) * D;          // D is a multiple of 8
    if ((reinterpret_cast<size_t>(src) & 15) == 0) {                     // 16-byte loads (1024 tokens of 2048, two rows each: 9.4 -> 6.5 us)
        for (uint32_t k = 4 * threadIdx.x; k < D; k += 4 * blockDim.x) {
            const float4 v = *reinterpret_cast<const float4*>(x + k);
            uint2 o;
            asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(o.x) : "f"(v.y), "f"(v.x));
            asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(o.y) : "f"(v.w), "f"(v.z));
            *reinterpret_cast<uint2*>(xs + ((size_t)r * D + k) / 2) = o;
        }
        return;
    }
    for (uint32_t k = 2 * threadIdx.x; k < D; k += 2 * blockDim.x) {
        uint32_t v;
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(v) : "f"(x[k + 1]), "f"(x[k]));
        xs[((size_t)r * D + k) / 2] = v;
    }
}
__global__ void k_moe_combine(float* __restrict__ dst, const float* __restrict__ src, const float* __restrict__ z, const float* __restrict__ route,
                              const int* __restrict__ pos_of_pair, uint32_t D, uint32_t top) {
    pdl_enter();
    const uint32_t t = blockIdx.x;
    if (((reinterpret_cast<size_t>(dst) | reinterpret_cast<size_t>(src)) & 15) == 0) {      // 16 bytes at a time, the same sums (11.5 -> 8 us)
        for (uint32_t d = 4 * threadIdx.x; d < D; d += 4 * blockDim.x) {
            float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 2
            for (uint32_t c = 0; c < top; c++) {
                const size_t pair = (size_t)t * top + c;
                const int pos = pos_of_pair[pair];
                const float w = route[2 * pair + 1];
                const float4 v = *reinterpret_cast<const float4*>((pos >= 0 ? z + (size_t)pos * D : src + (size_t)t * D) + d);
                acc = make_float4(fmaf(w, v.x, acc.x), fmaf(w, v.y, acc.y), fmaf(w, v.z, acc.z), fmaf(w, v.w, acc.w));
            }
            *reinterpret_cast<float4*>(dst + (size_t)t * D + d) = acc;
        }
        return;
    }
    for (uint32_t d = threadIdx.x; d < D; d += blockDim.x) {
        float acc = 0.0f;
        for (uint32_t c = 0; c < top; c++) {
            const size_t pair = (size_t)t * top + c;
            const int pos = pos_of_pair[pair];
            acc = fmaf(route[2 * pair + 1], pos >= 0 ? z[(size_t)pos * D + d] : src[(size_t)t * D + d], acc);
        }
        dst[(size_t)t * D + d] = acc;
    }
}

}  // namespace

static bool dense_gemm_enabled() {
    static const bool enabled = [] { const char* e = getenv("ZG_DENSE_GEMM"); return !(e && e[0] == '0'); }();
    return enabled;
}
// MOE_FFN on bfloat16 weights with enough (token, choice) pairs to fill tiles runs grouped on the tensor cores
static bool moe_grouped(const ZgSeqOp& s, float* const* bufs) {
    const uint32_t T = s.n[0], D = s.n[1], ff = s.n[2], E = s.n[3], top = s.n[4];
    if (!dense_gemm_enabled() || s.n[5] != ZG_W_BF16 || !E || E > kMoeMaxExperts || T * top <= 16 || D < 64 || ff < 64 || D % 8 || ff % 8) return false;
    if (!bufs) return true;
    for (int i = 0; i < 3; i++) if (reinterpret_cast<uintptr_t>(wptr<bf16>(bufs, s.buf[3], s.off[i])) & 15) return false;
    return true;
}
// f32 slots the op's own scratch operand (MOE_FFN buf[4]) must have; 0 for ops without one
size_t zg_seq_op_operand_scratch(const ZgOp& op) {
    if (op.tag != ZG_OP_MOE_FFN) return 0;
    const ZgSeqOp& s = op.u.seq;
    size_t n = (size_t)s.n[0] * s.n[4] * s.n[2];
    if (moe_grouped(s, nullptr)) { const size_t g = moe_layout(s.n[0], s.n[1], s.n[2], s.n[3], s.n[4]).total; if (g > n) n = g; }
    return n ? n : 1;
}
extern "C" __attribute__((visibility("default"))) size_t zg_cuda_seq_scratch_elems(const ZgOp* op) { return op ? zg_seq_op_operand_scratch(*op) : 0; }

uint32_t zg_delta_row_slices(uint32_t dim) {
    uint32_t rs = 1;
    while (rs * kDeltaRows < dim) rs <<= 1;
    return rs;
}

// Static checks of a sequence op against the program's buffer sizes (f32 slots): shapes, strides and every extent.
bool zg_seq_op_valid(const ZgOp& op, const size_t* elems, size_t n_bufs, char* why, size_t why_n) {
    if (op.tag >= ZG_OP_STREAM_STEP) return zg_stream_op_valid(op, elems, n_bufs, why, why_n);
    if (op.tag >= ZG_OP_SSM_SCAN) return zg_rec_op_valid(op, elems, n_bufs, why, why_n);
    if (op.tag >= ZG_OP_TOKEN_SHIFT) return zg_mix_op_valid(op, elems, n_bufs, why, why_n);
    const ZgSeqOp& s = op.u.seq;
    auto fail = [&](const char* m) { snprintf(why, why_n, "%s", m); return false; };
    auto have = [&](int i) { return s.buf[i] != ZG_NO_BUF && s.buf[i] < n_bufs; };
    auto fits = [&](int i, size_t off, size_t n) { return have(i) && off + n <= elems[s.buf[i]]; };
    const uint32_t wdt_of[] = {s.n[2], s.n[5], s.n[3], 0, s.n[6], s.n[9], s.n[4], s.n[5]};
    const uint32_t wdt = wdt_of[op.tag - ZG_OP_EMBED];
    if (wdt > ZG_W_BF16) return fail("unknown weight type");
    auto wfits = [&](int i, size_t off, size_t n) { return have(i) && (wdt == ZG_W_BF16 ? (off + n + 1) / 2 : off + n) <= elems[s.buf[i]]; };
    switch (op.tag) {
        case ZG_OP_EMBED: {
            const size_t T = s.n[0], D = s.n[1];
            if (!fits(0, 0, T * D) || !fits(1, ZG_CTL_IDS, T) || !have(2)) return fail("embed: extent");
            if (s.n[4] && (s.n[3] || s.n[5] >= s.n[4] || s.n[6] >= s.n[4] || !wfits(2, s.off[2], ((size_t)s.n[4] + 1) * D))) return fail("embed: bigram table");
            if (s.n[7] > 1 || (s.n[7] && !wfits(2, s.off[3], 2 * D + 1))) return fail("embed: norm");
            return true;
        }
        case ZG_OP_LINEAR: {
            const size_t M = s.n[0], N = s.n[1], K = s.n[2], srs = s.n[3], drs = s.n[4];
            if (!M || !N || !K || srs < K || drs < N) return fail("linear: shape");
            if (!fits(0, s.off[3], (M - 1) * drs + N) || !fits(1, s.off[2], (M - 1) * srs + K) || !wfits(2, s.off[0], (s.n[10] ? 2 : 1) * N * K)) return fail("linear: extent");
            if (s.n[10] > 1 || (s.n[10] && (s.buf[3] != ZG_NO_BUF || s.n[8] || s.n[9]))) return fail("linear: pairs take no bias and no column range");
            if (s.n[11] && !s.n[7]) return fail("linear: a row limit needs the rows of a state buffer");
            if (s.buf[3] != ZG_NO_BUF && !wfits(3, s.off[1], N)) return fail("linear: bias extent");
            if (s.buf[0] == s.buf[1]) return fail("linear: in place");
            if (s.n[6] > 6 || (s.n[6] == 5 && !(s.f[0] > 0.0f))) return fail("linear: activation");
            if (s.n[9] > N || s.n[8] > (s.n[9] ? s.n[9] : N)) return fail("linear: activation columns");
            if (s.n[7] && (s.n[7] < s.off[2] + (M - 1) * srs + K || !fits(4, 0, ZG_CTL_IDS))) return fail("linear: source slots");
            return true;
        }
        case ZG_OP_NORM: {
            const size_t n = (size_t)s.n[0] * s.n[1];
            auto bad_kind = [](uint32_t k) { return k > 63 || (k & 24u) == 24u || ((k & 32u) && (k & 24u)); };
            auto weights = [&](uint32_t k) { return (k & 8u) ? 2 * (size_t)s.n[1] + 1 : ((k & 32u) ? (size_t)1 : (size_t)s.n[1]); };
            if (!n || bad_kind(s.n[2])) return fail("norm: shape");
            const size_t w_need = weights(s.n[2]);      // Dynamic Tanh: weight, bias and alpha
            if (!fits(0, s.off[3], n) || !fits(1, 0, n) || (!(s.n[2] & 16u) && !wfits(2, s.off[0], w_need))) return fail("norm: extent");
            if (s.n[7]) {      // a second source, normed like the first with its own weight (off 2 of w's arena) and added to it
                if (s.n[7] > 1 || (s.n[2] & 24u) || s.n[5] || !fits(6, 0, n) || !wfits(2, s.off[2], w_need) || s.buf[6] == s.buf[0] || (s.buf[4] != ZG_NO_BUF && s.buf[6] == s.buf[4]))
                    return fail("norm: second source");
            } else if (((s.n[2] | (s.buf[4] != ZG_NO_BUF && !s.n[5] ? s.n[4] : 0u)) & 24u) && (s.n[5] || s.buf[6] != ZG_NO_BUF))
                return fail("norm: kinds without statistics take no averaged source and no token shift");
            if (s.n[8]) {      // an outer norm over the (sum of the) normed source(s)
                const uint32_t ko = s.n[8] - 1;
                if (bad_kind(ko) || (ko & 28u) || (s.n[2] & 24u) || s.n[5] || (!s.n[7] && s.buf[6] != ZG_NO_BUF) || !wfits(2, s.off[5], weights(ko)) || s.buf[0] == s.buf[3])
                    return fail("norm: outer norm");
            }
            if (s.n[5]) {      // averaged source
                if (s.n[6] < n || !fits(1, 0, (size_t)(s.n[5] - 1) * s.n[6] + n) || !wfits(2, s.off[4], s.n[5]) || s.buf[3] != ZG_NO_BUF || !fits(4, 0, n) || s.buf[4] == s.buf[0] ||
                    s.buf[4] == s.buf[1])
                    return fail("norm: averaged source");
                if (s.buf[6] != ZG_NO_BUF && (s.n[0] != 1 || !have(6) || elems[s.buf[6]] < s.n[1] || !wfits(2, s.off[2], s.n[1]) || !fits(7, 0, ZG_CTL_IDS))) return fail("norm: fused token shift (single-row steps)");
                return true;
            }
            if (s.buf[3] != ZG_NO_BUF && !fits(3, 0, n)) return fail("norm: residual extent");
            if (s.buf[4] != ZG_NO_BUF && (bad_kind(s.n[4]) || !fits(4, 0, n) || (!(s.n[4] & 16u) && !wfits(5, s.off[1], weights(s.n[4]))) || s.buf[4] == s.buf[0] || s.buf[4] == s.buf[1] || s.buf[4] == s.buf[3]))
                return fail("norm: chained norm");
            if (!s.n[7] && s.buf[6] != ZG_NO_BUF && (s.n[0] != 1 || !have(6) || elems[s.buf[6]] < s.n[1] || !wfits(s.buf[4] != ZG_NO_BUF ? 5 : 2, s.off[2], s.n[1]) || !fits(7, 0, ZG_CTL_IDS)))
                return fail("norm: fused token shift (single-row steps)");
            return true;
        }
        case ZG_OP_WINDOW_ATTENTION: {
            const size_t T = s.n[0], H = s.n[1], G = s.n[2], dim = s.n[3], rs = s.n[4], win = s.n[5], R = s.n[6];
            if (!T || !H || !G || H % G || !dim || dim > kAttnMaxDim || !win || R < win - 1 + T) return fail("window_attention: shape");
            if (s.off[0] + H * dim > rs || s.off[1] + G * dim > rs || s.off[2] + H * dim > rs) return fail("window_attention: columns");
            if (!fits(0, 0, T * H * dim) || !fits(1, 0, T * rs) || !have(2) || elems[s.buf[2]] < R * G * dim || !fits(3, 0, win * H) || !fits(4, 0, ZG_CTL_IDS))
                return fail("window_attention: extent");
            return true;
        }
        case ZG_OP_CAUSAL_CONV: {
            const size_t T = s.n[0], C = s.n[1], taps = s.n[2], srs = s.n[3], drs = s.n[4];
            if (!T || !C || taps < 1 || srs < C || drs < C || s.n[5] > 1) return fail("causal_conv: shape");
            if (!fits(0, s.off[2], (T - 1) * drs + C) || !fits(1, s.off[1], (T - 1) * srs + C) || !wfits(2, s.off[0], C * taps) || !have(3) || !fits(4, 0, ZG_CTL_IDS))
                return fail("causal_conv: extent");
            if (taps > 1 && elems[s.buf[3]] < (taps - 1) * C) return fail("causal_conv: state size");
            if (s.n[7] > 1 || (s.n[7] && !wfits(2, s.off[3], C))) return fail("causal_conv: bias");
            if (s.buf[0] == s.buf[1]) return fail("causal_conv: in place");
            return true;
        }
        case ZG_OP_DELTA_RULE: {
            const size_t T = s.n[0], H = s.n[1], G = s.n[2], dim = s.n[3], vdim = s.n[4];
            const size_t form = s.n[10], drs = s.n[11] ? s.n[11] : H * vdim;
            if (!T || !H || !G || H % G || !dim || !vdim || zg_delta_row_slices((uint32_t)dim) > 32 || form > 255) return fail("delta_rule: shape");
            if (((form & 32) && (!(form & 1) || !wfits(5, s.n[14], H * dim))) || (form & 66) == 66) return fail("delta_rule: bonus or decay form");
            if (s.n[12] + H * vdim > drs || ((form & 2) && !(s.f[3] > 0.0f))) return fail("delta_rule: form");
            if (s.off[0] + G * dim > s.n[5] || s.off[1] + G * dim > s.n[5] || s.off[2] + H * vdim > s.n[5] || (!(form & 1) && s.off[3] + H > s.n[6]) || s.n[13] + H * (form & 16 ? 1 : dim) > s.n[7] || s.off[7] + H * vdim > s.n[8])
                return fail("delta_rule: columns");
            if (!fits(0, 0, (T - 1) * drs + s.n[12] + H * vdim) || !fits(1, 0, T * s.n[5]) || (!(form & 1) && !fits(2, 0, T * s.n[6])) || !fits(3, 0, T * s.n[7]) || !fits(4, 0, T * s.n[8]) ||
                (!(form & 66) && !wfits(5, s.off[4], H)) || !wfits(5, s.off[5], H * (form & 16 ? 1 : dim)) || !wfits(5, s.off[6], form & 128 ? H * vdim : vdim) || !have(6) || elems[s.buf[6]] < H * dim * vdim || !fits(7, 0, ZG_CTL_IDS))
                return fail("delta_rule: extent");
            return true;
        }
        case ZG_OP_ROUTE: {
            const size_t T = s.n[0], NE = s.n[1], top = s.n[2], rs = s.n[3];
            if (!T || !NE || !top || top > NE || rs < NE || NE > 4096 || s.n[5] > 3) return fail("route: shape");
            if (s.n[5] >= 2 && s.n[6] > 1 && (NE % s.n[6] || s.n[6] > 1024 || !s.n[7] || s.n[7] > s.n[6] || (size_t)s.n[7] * (NE / s.n[6]) < top)) return fail("route: groups");
            if (!fits(0, 0, T * top * 2) || !fits(1, s.off[1], (T - 1) * rs + NE) || !wfits(2, s.off[0], NE)) return fail("route: extent");
            return true;
        }
        case ZG_OP_MOE_FFN: {
            const size_t T = s.n[0], D = s.n[1], ff = s.n[2], E = s.n[3], top = s.n[4];
            if (!T || !D || !top) return fail("moe_ffn: shape");
            if (!fits(0, 0, T * D) || !fits(1, 0, T * D) || !fits(2, 0, T * top * 2) || !fits(4, 0, zg_seq_op_operand_scratch(op)) ||
                (E && (!wfits(3, s.off[0], E * ff * D) || !wfits(3, s.off[1], E * ff * D) || !wfits(3, s.off[2], E * ff * D))))
                return fail("moe_ffn: extent");
            if (s.buf[0] == s.buf[1]) return fail("moe_ffn: in place");
            return true;
        }
        default: return fail("not a sequence op");
    }
}

// which of buf[0..8) an op writes (bit i); everything else it names is read
uint32_t zg_seq_op_writes(uint32_t tag) {
    switch (tag) {
        case ZG_OP_NORM: return 1u | (1u << 4) | (1u << 6);   // a chained second destination and a token-shift state, when named
        case ZG_OP_WINDOW_ATTENTION: return 1u | (1u << 2);
        case ZG_OP_CAUSAL_CONV: return 1u | (1u << 3);
        case ZG_OP_DELTA_RULE: return 1u | (1u << 6);
        case ZG_OP_MOE_FFN: return 1u | (1u << 4);
        case ZG_OP_STREAM_STEP: return 1u | (1u << 5) | (1u << 6);   // streams, the next sublayer's input, a carried row
        default: return tag >= ZG_OP_SSM_SCAN ? zg_rec_op_writes(tag) : (tag >= ZG_OP_TOKEN_SHIFT ? zg_mix_op_writes(tag) : 1u);
    }
}

// f32 slots of the shared activation scratch this op needs (0: none): a LINEAR over bfloat16 weights with more rows than the
// row kernels take runs on the tensor cores (dense_gemm.cu) from a bf16 copy of its input.  ZG_DENSE_GEMM=0 keeps the exact tile.
// window shares per (token, head) of a WINDOW_ATTENTION step: few pairs and a long window (decode) spread over more CTAs
static uint32_t attention_splits(const ZgSeqOp& s) {
    const uint32_t pairs = s.n[0] * s.n[1], window = s.n[5];
    if (s.n[3] % 4 || pairs >= 128 || window < 128 || (s.n[0] >= (uint32_t)kWaTiledMinTokens && s.n[3] <= 128)) return 1;   // the tiled prefill kernel splits nothing
    uint32_t S = (256 + pairs - 1) / pairs;
    if (S > window / 32) S = window / 32;
    return S < 2 ? 1 : (S > 16 ? 16 : S);
}
static bool linear_split(const ZgSeqOp& s, float* const* bufs) {     // f32 weights, many rows: split operands on the tensor cores
    return zg_split_gemm_usable(wptr<float>(bufs, s.buf[2], s.off[0]), bufs[s.buf[1]] + s.off[2], s.n[0], s.n[10] ? 2 * s.n[1] : s.n[1], s.n[2], s.n[3], s.n[7]);
}
unsigned int zg_seq_timeouts() { return tc_timeouts(); }
size_t zg_seq_op_scratch_elems(const ZgOp& op, float* const* bufs, bool least) {
    if (op.tag >= ZG_OP_STREAM_STEP) return 0;
    if (op.tag >= ZG_OP_SSM_SCAN) return zg_rec_op_scratch_elems(op);
    if (op.tag >= ZG_OP_TOKEN_SHIFT) return zg_mix_op_scratch_elems(op);
    if (op.tag == ZG_OP_WINDOW_ATTENTION) {
        const uint32_t S = attention_splits(op.u.seq);
        return S > 1 ? (size_t)op.u.seq.n[0] * op.u.seq.n[1] * S * (4 + op.u.seq.n[3]) : 0;
    }
    if (op.tag == ZG_OP_DELTA_RULE) {                  // the prepared per-token rows of the prefill form
        const ZgSeqOp& d = op.u.seq;
        if (d.n[0] < (uint32_t)kDeltaPrepMinTokens || d.n[3] > kWalkMaxDim) return 0;
        const bool plain = d.n[10] & kDeltaPlain;
        if (delta_by_blocks(d.n[0], d.n[1], d.n[3], d.n[4])) return (size_t)((d.n[0] + kBlockTokens - 1) / kBlockTokens) * d.n[1] * delta_block_elems(32 * delta_block_rows(d.n[3]), plain);
        return delta_chunk_elems(delta_rows(d.n[3]), plain, d.n[4]) * d.n[1] * delta_pass_chunks(d.n[0], d.n[1], d.n[3], d.n[4], plain);
    }
    if (!dense_gemm_enabled() || op.tag != ZG_OP_LINEAR) return 0;
    const ZgSeqOp& s = op.u.seq;
    if (s.n[5] == ZG_W_F32) return linear_split(s, bufs) ? zg_split_gemm_scratch_elems(s.n[0], s.n[10] ? 2 * s.n[1] : s.n[1], s.n[2], least) : 0;
    if (!zg_dense_gemm_usable(wptr<bf16>(bufs, s.buf[2], s.off[0]), s.n[0], s.n[10] ? 2 * s.n[1] : s.n[1], s.n[2])) return 0;
    return zg_dense_gemm_scratch_elems(s.n[0], s.n[2]);
}

// Below that, a warp per output row and no staging is faster (four feed-forwards of 256 / 512, one row 27 us against 33; two rows 35 against 39, of 256 / 1024 44 against
// 39).  Pairs whose outputs are one wave of such warps need half as much again (gated feed-forwards of 512 / 1024, bfloat16, one row, 2 MB: 8.7 us each against 9.6;
// 256 / 1024, four rows, 1 MB: 17.2 against 22.0; 384 / 1024, one row 9.2 both ways, four rows, 1.5 MB: 20.0 against 14.9).
static bool linear_ring(uint32_t M, uint32_t N, bool pairs, size_t weight_bytes) {
    const size_t least = M == 1 ? 3u << 19 : 3u << 18;
    return weight_bytes >= (pairs && N <= 8 * zg_sm_count() ? least * 3 / 2 : least);
}
template <typename WT, bool PAIRS>
static bool launch_linear_ring(float* dst, const float* src, const WT* W, const WT* bias, uint32_t M, uint32_t N, uint32_t K, uint32_t src_rs, uint32_t dst_rs, SeqAct act,
                               const float* ctl, uint32_t slot_stride, bool early, const RingPlan& r, cudaStream_t st) {
#define ZG_RING(MR_, SPLIT_)                                                                                                                                  \
    do {                                                                                                                                                      \
        if (!zg_smem_limit<k_linear_rows_ring<WT, MR_, PAIRS, SPLIT_>>(kRingSmem)) return false;                                                              \
        launch_pdl(k_linear_rows_ring<WT, MR_, PAIRS, SPLIT_>, dim3(r.ctas), dim3(288), r.smem, st, dst, src, W, bias, M, N, K, src_rs, dst_rs, act, ctl,     \
                   slot_stride, r.lanes, r.segment, r.rows, early ? 1u : 0u);                                                                                 \
    } while (0)
    if (M == 1) ZG_RING(1, false); else if (M == 2) ZG_RING(2, false);
    else if (r.split) { if (M <= 4) ZG_RING(4, true); else ZG_RING(8, true); }
    else if (M <= 4) ZG_RING(4, false); else ZG_RING(8, false);
#undef ZG_RING
    return true;
}
bool zg_launch_seq_op(ZgCudaCtx* ctx, const ZgOp& op, float* const* bufs, float* scratch, size_t scratch_elems, cudaStream_t st, bool ahead) {
    (void)ctx;
    const ZgSeqOp& s = op.u.seq;
    switch (op.tag) {
        case ZG_OP_EMBED:
            ZG_SEQ_WDT(s.n[2], launch_pdl(k_embed<WT>, dim3(s.n[0], (s.n[1] + 255) / 256), dim3(256), 0, st, bufs[s.buf[0]], bufs[s.buf[1]], wptr<WT>(bufs, s.buf[2], s.off[0]), s.n[1], s.f[0],
                                          s.n[3] ? wptr<WT>(bufs, s.buf[2], s.off[1]) : nullptr, s.n[4] ? wptr<WT>(bufs, s.buf[2], s.off[2]) : nullptr, s.n[4], s.n[5], s.n[6],
                                          s.n[7] ? wptr<WT>(bufs, s.buf[2], s.off[3]) : nullptr));
            ZG_SEQ_CHECK();
            return true;
        case ZG_OP_LINEAR: {
            const uint32_t M = s.n[0], N = s.n[1], K = s.n[2];
            float* dst = bufs[s.buf[0]] + s.off[3];
            const float* src = bufs[s.buf[1]] + s.off[2];
            const bool has_bias = s.buf[3] != ZG_NO_BUF;
            const bool pairs = s.n[10] != 0;
            const SeqAct act = {s.n[6], s.f[0], s.n[8], s.n[9] ? s.n[9] : N};
            const float* slot_ctl = s.n[7] ? (const float*)bufs[s.buf[4]] : (const float*)nullptr;      // the source is the slot's part of a state buffer
            if (scratch && s.n[5] == ZG_W_F32 && zg_seq_op_scratch_elems(op, bufs))
                return zg_split_gemm_launch(wptr<float>(bufs, s.buf[2], s.off[0]), has_bias ? wptr<float>(bufs, s.buf[3], s.off[1]) : nullptr, src, dst, M, pairs ? 2 * N : N, K,
                                            s.n[3], s.n[4], scratch, scratch_elems, st, s.n[6], s.f[0], act.lo, act.hi, slot_ctl, s.n[7], pairs, s.n[11]);
            if (scratch && zg_seq_op_scratch_elems(op, bufs))
                return zg_dense_gemm_launch(wptr<bf16>(bufs, s.buf[2], s.off[0]), has_bias ? wptr<bf16>(bufs, s.buf[3], s.off[1]) : nullptr, src, dst, M, N, K,
                                            s.n[3], s.n[4], scratch, st, s.n[6], s.f[0], act.lo, act.hi, slot_ctl, s.n[7], pairs, s.n[11]);
#define ZG_ROWS(PAIRS_)                                                                                                                              \
    do {                                                                                                                                             \
        if (vec && M == 1) launch_pdl(k_linear_rows_vec<WT, 1, PAIRS_>, dim3(grid), dim3(256), xs_bytes, st, dst, src, W, b, M, N, K, s.n[3], s.n[4], act, slot_ctl, s.n[7]);      \
        else if (vec && M <= 4) launch_pdl(k_linear_rows_vec<WT, 4, PAIRS_>, dim3(grid), dim3(256), xs_bytes, st, dst, src, W, b, M, N, K, s.n[3], s.n[4], act, slot_ctl, s.n[7]); \
        else if (vec) launch_pdl(k_linear_rows_vec<WT, 8, PAIRS_>, dim3(grid), dim3(256), xs_bytes, st, dst, src, W, b, M, N, K, s.n[3], s.n[4], act, slot_ctl, s.n[7]);           \
        else launch_pdl(k_linear_rows<WT, PAIRS_>, dim3(grid), dim3(256), 0, st, dst, src, W, b, M, N, K, s.n[3], s.n[4], act, slot_ctl, s.n[7]);                                  \
    } while (0)
            ZG_SEQ_WDT(s.n[5], {
                const WT* W = wptr<WT>(bufs, s.buf[2], s.off[0]);
                const WT* b = has_bias ? wptr<WT>(bufs, s.buf[3], s.off[1]) : nullptr;
                constexpr uint32_t V = WVec<WT>::n;
                if (M <= kGemvRows) {
                    const size_t xs_bytes = (size_t)M * K * sizeof(float);
                    const bool aligned = K % V == 0 && (reinterpret_cast<size_t>(W) & 15) == 0, vec = aligned && xs_bytes <= 48 * 1024;
                    const dim3 grid((N + 7) / 8);
                    const RingPlan ring = ring_plan(M, N, K, pairs, sizeof(WT), zg_sm_count());
                    if (aligned && ring.smem && linear_ring(M, N, pairs, (size_t)(pairs ? 2 : 1) * N * K * sizeof(WT))) {
                        if (!(pairs ? launch_linear_ring<WT, true> : launch_linear_ring<WT, false>)(dst, src, W, b, M, N, K, s.n[3], s.n[4], act, slot_ctl, s.n[7], ahead, ring, st)) return false;
                        ZG_SEQ_CHECK();
                        return true;
                    }
                    if (pairs) ZG_ROWS(true); else ZG_ROWS(false);
                } else {
                    const uint32_t NW = pairs ? 2 * N : N;
                    const dim3 grid((NW + kTN - 1) / kTN, (M + kTM - 1) / kTM);
                    if (pairs) k_linear_tile<WT, true><<<grid, 256, 0, st>>>(dst, src, W, b, M, NW, K, s.n[3], s.n[4], act, slot_ctl, s.n[7], s.n[11]);
                    else k_linear_tile<WT, false><<<grid, 256, 0, st>>>(dst, src, W, b, M, NW, K, s.n[3], s.n[4], act, slot_ctl, s.n[7], s.n[11]);
                }
            });
#undef ZG_ROWS
            ZG_SEQ_CHECK();
            return true;
        }
        case ZG_OP_NORM: {
            const float* res = s.buf[3] != ZG_NO_BUF ? bufs[s.buf[3]] : nullptr;
            float* dst2 = s.buf[4] != ZG_NO_BUF ? bufs[s.buf[4]] : nullptr;
            float* shift_state = s.buf[6] != ZG_NO_BUF ? bufs[s.buf[6]] : nullptr;
            const uint32_t avg_terms = s.n[5];             // averaged source: buf 4 receives the average instead of a chained norm
            if (((s.n[2] | (dst2 ? s.n[4] : 0u)) & 24u) || s.n[7] || s.n[8]) {   // Dynamic Tanh or the plain residual step somewhere in the launch, or two sources
#define ZG_NORM_ANY(KEEP_, THREADS_)                                                                                                               \
    ZG_SEQ_WDT(s.n[3], launch_pdl(k_norm_any<WT, KEEP_, THREADS_>, dim3(s.n[0]), dim3(THREADS_), 0, st, bufs[s.buf[0]] + s.off[3], (const float*)bufs[s.buf[1]], \
                                  (s.n[2] & 16u) ? (const WT*)nullptr : wptr<WT>(bufs, s.buf[2], s.off[0]), res, s.n[1], s.n[2], s.f[0], dst2,                \
                                  dst2 && !(s.n[4] & 16u) ? wptr<WT>(bufs, s.buf[5], s.off[1]) : (const WT*)nullptr, s.n[4], s.f[1],                         \
                                  s.n[7] ? (const float*)bufs[s.buf[6]] : (const float*)nullptr, s.n[7] ? wptr<WT>(bufs, s.buf[2], s.off[2]) : (const WT*)nullptr, \
                                  s.n[8] ? s.n[8] - 1 : 0u, s.n[8] ? wptr<WT>(bufs, s.buf[2], s.off[5]) : (const WT*)nullptr, ahead && s.n[0] < 64))
                // Many rows: the kernel that keeps a row in registers (64 each: 1024 threads an SM) as long as all rows are resident at once.  Each value is then read once
                // and all its loads are in flight together; the other one walks a row up to four times.  Feed-forwards of f32 / bf16 weights, walked -> in registers:
                // 64 tokens of 4096 101.4 -> 91.8 / 68.2 -> 63.6 us, 256 of 2048 97.3 -> 92.3 / 53.3 -> 52.2, 256 of 1024 46.9 -> 45.3 / 36.9 -> 34.9.  Up to 512 columns
                // two values a thread leave nothing to overlap (300 of 512: 37.0 -> 38.6), and past one wave a second one begins where the walk has 2048 threads an SM.
                // Their weights are read after the wait, as the walk reads them.
                const uint32_t cols = s.n[1], resident = zg_sm_count() * (cols <= 1024 ? 4u : cols <= 2048 ? 2u : 1u);
                if (cols > 4096 || (s.n[0] >= 64 && (cols <= 512 || s.n[0] > resident)))
                    ZG_SEQ_WDT(s.n[3], launch_pdl(k_norm_any_rows<WT>, dim3(s.n[0]), dim3(256), 0, st, bufs[s.buf[0]] + s.off[3], (const float*)bufs[s.buf[1]],
                                                  (s.n[2] & 16u) ? (const WT*)nullptr : wptr<WT>(bufs, s.buf[2], s.off[0]), res, s.n[1], s.n[2], s.f[0], dst2,
                                                  dst2 && !(s.n[4] & 16u) ? wptr<WT>(bufs, s.buf[5], s.off[1]) : (const WT*)nullptr, s.n[4], s.f[1],
                                                  s.n[7] ? (const float*)bufs[s.buf[6]] : (const float*)nullptr, s.n[7] ? wptr<WT>(bufs, s.buf[2], s.off[2]) : (const WT*)nullptr,
                                                  s.n[8] ? s.n[8] - 1 : 0u, s.n[8] ? wptr<WT>(bufs, s.buf[2], s.off[5]) : (const WT*)nullptr));
                // Four values a thread: with eight the unrolled code is twice as long and each launch fetches it anew (four feed-forwards of one token, 2048 / 4096,
                // whose 2048 columns had 256 threads: 88 us, with 512 threads 76, with 1024 of two values 80).
                else if (s.n[1] <= 1024) ZG_NORM_ANY(4, 256);
                else if (s.n[1] <= 2048) ZG_NORM_ANY(4, 512);
                // Up to 4096 columns in registers (eight values and 512 threads / four and 1024, per launch in a chain: 2056 columns 3.39 / 2.82 us, 4096 4.03 / 3.07, two sources
                // of 4096 5.16 / 4.61; four feed-forwards of 2304 / 6912 136 / 121); wider rows are walked from memory.
                else ZG_NORM_ANY(4, 1024);
#undef ZG_NORM_ANY
                ZG_SEQ_CHECK();
                return true;
            }
            if (avg_terms) dst2 = nullptr;
            ZG_SEQ_WDT(s.n[3], launch_pdl(k_norm<WT>, dim3(s.n[0]), dim3(256), 0, st, bufs[s.buf[0]] + s.off[3], bufs[s.buf[1]], wptr<WT>(bufs, s.buf[2], s.off[0]), res, s.n[1], s.n[2], s.f[0],
                                          dst2, dst2 ? wptr<WT>(bufs, s.buf[5], s.off[1]) : nullptr, s.n[4], s.f[1],
                                          shift_state ? wptr<WT>(bufs, s.buf[dst2 ? 5 : 2], s.off[2]) : nullptr, shift_state, shift_state ? bufs[s.buf[7]] : nullptr,
                                          avg_terms ? wptr<WT>(bufs, s.buf[2], s.off[4]) : nullptr, avg_terms, s.n[6], avg_terms ? bufs[s.buf[4]] : nullptr, ahead));
            ZG_SEQ_CHECK();
            return true;
        }
        case ZG_OP_WINDOW_ATTENTION: {
            const uint32_t T = s.n[0], H = s.n[1], G = s.n[2], dim = s.n[3];
            launch_pdl(k_ring_append, dim3(T), dim3(128), 0, st, bufs[s.buf[2]], bufs[s.buf[1]], bufs[s.buf[4]], s.off[1], s.n[4], G * dim, s.n[6]);
            ZG_SEQ_CHECK();
            const size_t width = (size_t)G * dim;
            const bool vec = dim % 4 == 0 && s.off[0] % 4 == 0 && s.n[4] % 4 == 0 && width % 4 == 0 && (reinterpret_cast<uintptr_t>(bufs[s.buf[1]]) & 15) == 0 &&
                             (reinterpret_cast<uintptr_t>(bufs[s.buf[2]]) & 15) == 0;
            if (vec && s.off[2] % 4 == 0 && T >= kWaTiledMinTokens && dim <= 128) {
                switch ((dim + 15) / 16) {
                    case 1: launch_window_attention_tiled<1>(s, bufs, st); break;
                    case 2: launch_window_attention_tiled<2>(s, bufs, st); break;
                    case 3: launch_window_attention_tiled<3>(s, bufs, st); break;
                    case 4: launch_window_attention_tiled<4>(s, bufs, st); break;
                    case 5: launch_window_attention_tiled<5>(s, bufs, st); break;
                    case 6: launch_window_attention_tiled<6>(s, bufs, st); break;
                    case 7: launch_window_attention_tiled<7>(s, bufs, st); break;
                    default: launch_window_attention_tiled<8>(s, bufs, st); break;
                }
            } else if (vec) {
                const uint32_t CH = dim > 128 ? 2 : 1;
                uint32_t LK = 1;
                while (LK * 4 * CH < dim) LK <<= 1;
                const uint32_t S = scratch ? attention_splits(s) : 1;
                float* part = S > 1 ? scratch : nullptr;
                const uint32_t nw = S > 1 ? 4 : (T * H <= 64 ? 16 : (T * H <= 1024 ? 8 : 4));
                const size_t smem = (size_t)nw * (4 + dim) * sizeof(float);
                if (CH == 1)
                    launch_pdl(k_window_attention_v<1>, dim3(T * H, S), dim3(nw * 32), smem, st, bufs[s.buf[0]], bufs[s.buf[1]], bufs[s.buf[2]], bufs[s.buf[3]], bufs[s.buf[4]], H, G, dim, LK,
                                                                        s.n[4], s.off[0], s.off[2], s.n[5], s.n[6], s.f[0], s.f[1], part);
                else
                    launch_pdl(k_window_attention_v<2>, dim3(T * H, S), dim3(nw * 32), smem, st, bufs[s.buf[0]], bufs[s.buf[1]], bufs[s.buf[2]], bufs[s.buf[3]], bufs[s.buf[4]], H, G, dim, LK,
                                                                        s.n[4], s.off[0], s.off[2], s.n[5], s.n[6], s.f[0], s.f[1], part);
                if (S > 1) {
                    ZG_SEQ_CHECK();
                    launch_pdl(k_window_attention_merge, dim3(T * H), dim3(128), 0, st, bufs[s.buf[0]], bufs[s.buf[1]], part, H, dim, S, s.n[4], s.off[2]);
                }
            } else {
                const uint32_t warps = 4;
                launch_pdl(k_window_attention, dim3((T * H + warps - 1) / warps), dim3(warps * 32), warps * dim * sizeof(float), st, 
                    bufs[s.buf[0]], bufs[s.buf[1]], bufs[s.buf[2]], bufs[s.buf[3]], bufs[s.buf[4]], T, H, G, dim, s.n[4], s.off[0], s.off[2], s.n[5], s.n[6], s.f[0], s.f[1]);
            }
            ZG_SEQ_CHECK();
            return true;
        }
        case ZG_OP_CAUSAL_CONV: {
            const uint32_t T = s.n[0], C = s.n[1], taps = s.n[2];
            float* dst = bufs[s.buf[0]] + s.off[2];
            const float* src = bufs[s.buf[1]] + s.off[1];
            const size_t n = (size_t)T * C;
            ZG_SEQ_WDT(s.n[6], launch_pdl(k_causal_conv<WT>, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st, dst, src, wptr<WT>(bufs, s.buf[2], s.off[0]), bufs[s.buf[3]], bufs[s.buf[4]],
                                                                                          T, C, taps, s.n[3], s.n[4], s.n[5], (uint32_t)(T == 1 && taps > 1),
                                                                                          s.n[7] ? wptr<WT>(bufs, s.buf[2], s.off[3]) : nullptr));
            ZG_SEQ_CHECK();
            if (taps > 1 && T > 1) {
                launch_pdl(k_conv_advance, dim3((C + 127) / 128), dim3(128), 0, st, bufs[s.buf[3]], src, bufs[s.buf[4]], T, C, taps, s.n[3]);
                ZG_SEQ_CHECK();
            }
            return true;
        }
        case ZG_OP_DELTA_RULE: {
            const uint32_t T = s.n[0], H = s.n[1], G = s.n[2], dim = s.n[3], vdim = s.n[4];
            const uint32_t form = s.n[10], dst_rs = s.n[11] ? s.n[11] : H * vdim;
            const float inv_tau = (form & kDeltaSigmoidDecay) ? 1.0f / s.f[3] : 0.0f, out_scale = (form & kDeltaOutScale) ? s.f[4] : 1.0f;
            float* dst = bufs[s.buf[0]] + s.n[12];
            const float* betab = (form & kDeltaPlain) ? nullptr : bufs[s.buf[2]];
            const uint32_t RS = zg_delta_row_slices(dim), cols = kDeltaThreads / RS;
            const size_t smem = ((size_t)3 * kDeltaTile * RS * kDeltaRows + kDeltaTile) * sizeof(float);
            const dim3 grid((vdim + cols - 1) / cols, H);
            if (scratch && T >= (uint32_t)kDeltaPrepMinTokens && delta_by_blocks(T, H, dim, vdim)) {
                const uint32_t R = delta_block_rows(dim), wcols = kBlockThreads / 32 * kBlockCols, n_prep = delta_block_prep_ctas(T, H);
                // Many CTAs: a plain launch.  CTAs placed while the predecessor still fills the GPU share SMs two by two.
                const bool plain = form & kDeltaPlain, early = n_prep + (vdim + wcols - 1) / wcols * H <= kBlockSideBySide;
#define ZG_BLOCK_FORM(R_, PLAIN_)                                                                                                                             \
    do {                                                                                                                                                      \
        constexpr size_t walk_smem = (size_t)2 * (kDeltaTile / kBlockTokens) * delta_block_elems(32 * R_, PLAIN_) * sizeof(float);                            \
        if (!zg_smem_limit<k_delta_block_walk<R_, PLAIN_>>(walk_smem)) return false;                                                                          \
        launch_pdl_if(early, k_delta_block_walk<R_, PLAIN_>, dim3((vdim + wcols - 1) / wcols, H), dim3(kBlockThreads), walk_smem, st, dst, bufs[s.buf[1]],    \
                      scratch, bufs[s.buf[6]], bufs[s.buf[7]], T, H, dim, vdim, s.off[2], s.n[5], dst_rs);                                                    \
    } while (0)
#define ZG_BLOCK(R_)                                                                                                                                          \
    do {                                                                                                                                                      \
        ZG_SEQ_WDT(s.n[9], launch_pdl(k_delta_block_prepare<WT, R_>, dim3(n_prep), dim3(128), 0, st, scratch, bufs[s.buf[1]], betab, bufs[s.buf[3]] + s.n[13], \
                                      wptr<WT>(bufs, s.buf[5], 0), T, H, G, dim, s.off[0], s.off[1], s.off[3], s.off[4], s.off[5], s.n[5], s.n[6], s.n[7],    \
                                      s.f[1], s.f[2], form, inv_tau, s.n[14]));                                                                               \
        ZG_SEQ_CHECK();                                                                                                                                       \
        if (plain) ZG_BLOCK_FORM(R_, true); else ZG_BLOCK_FORM(R_, false);                                                                                    \
    } while (0)
                if (R == 2) ZG_BLOCK(2); else ZG_BLOCK(4);
#undef ZG_BLOCK
#undef ZG_BLOCK_FORM
            } else if (scratch && T >= (uint32_t)kDeltaPrepMinTokens && dim <= kWalkMaxDim) {
                const bool plain = form & kDeltaPlain;
                const uint32_t dpad = delta_rows(dim), warps = dpad == 64 ? 4 : 8, pass = delta_pass_chunks(T, H, dim, vdim, plain) * kWalkChunk;
                // Where every CTA has an SM to itself: three stages, a chunk's vectors are asked for two chunks ahead, and more than half of the SM's shared
                // memory (two CTAs on one SM share what bounds them while other SMs stand idle).  Two stages and several CTAs per SM where there are more.
                const bool alone = (vdim + kWalkCols - 1) / kWalkCols * H <= zg_sm_count();
                const uint32_t stages = dpad == 512 ? 1 : alone ? kWalkStages : 2;
                const size_t walk_smem = std::max(delta_walk_smem(dpad, plain, warps, stages), alone ? kWalkAlone : 0u);
                ZG_SEQ_WDT(s.n[9], if (!zg_smem_limit<k_delta_prepare<WT>>(delta_prep_smem(kWalkMaxDim))) return false);
                for (uint32_t t = 0; t < T; t += pass) {
                    const uint32_t n = std::min(pass, T - t);
                    // Up to one CTA per SM: eight warps each, and the walk may be placed beside them; up to two where the walk has an SM per CTA or vectors are long
                    // (16 heads of 128 x 128, 160 tokens 29 us, with four warps and no early walk 39; 32 heads of 64 x 64, 80 tokens 18.5 and 23.5; but 40 heads, 112
                    // tokens 28.7 and 25.4).  More: four warps (1024 CTAs 41 us, with eight 47).
                    const uint32_t n_prep = (n + kWalkChunk - 1) / kWalkChunk * H;
                    const bool few = n_prep <= (alone || dpad > 64 ? 2 : 1) * zg_sm_count();
                    ZG_SEQ_WDT(s.n[9], launch_pdl(k_delta_prepare<WT>, dim3(H, n_prep / H), dim3(few ? kDeltaPrepThreads : kDeltaPrepThreads / 2), delta_prep_smem(dpad), st, scratch, bufs[s.buf[1]] + (size_t)t * s.n[5],
                                                  betab ? betab + (size_t)t * s.n[6] : nullptr, bufs[s.buf[3]] + s.n[13] + (size_t)t * s.n[7], wptr<WT>(bufs, s.buf[5], 0), n, H, G, dim, vdim, dpad,
                                                  s.off[0], s.off[1], s.off[2], s.off[3], s.off[4], s.off[5], s.n[5], s.n[6], s.n[7], s.f[1], s.f[2], form, inv_tau, s.n[14], few ? 1u : 0u));
                    ZG_SEQ_CHECK();
#define ZG_WALK(SL_, WARPS_, PLAIN_)                                                                                                                           \
    do {                                                                                                                                                      \
        constexpr uint32_t rows = 16 * SL_ * WARPS_, most = delta_walk_smem(rows, PLAIN_, WARPS_, rows == 512 ? 1 : kWalkStages);                             \
        if (!zg_smem_limit<k_delta_walk<SL_, WARPS_, PLAIN_>>(std::max(most, kWalkAlone))) return false;                                                      \
        launch_pdl(k_delta_walk<SL_, WARPS_, PLAIN_>, dim3((vdim + kWalkCols - 1) / kWalkCols, H), dim3(64 * WARPS_), walk_smem, st, dst + (size_t)t * dst_rs, \
                   scratch, bufs[s.buf[6]], bufs[s.buf[7]], n, H, dim, vdim, dst_rs, stages);                                                                 \
    } while (0)
#define ZG_WALK_ROWS(PLAIN_)                                                                                                                                   \
    do {                                                                                                                                                      \
        if (dpad == 512) ZG_WALK(4, 8, PLAIN_); else if (dpad == 256) ZG_WALK(2, 8, PLAIN_); else if (dpad == 128) ZG_WALK(1, 8, PLAIN_); else ZG_WALK(1, 4, PLAIN_); \
    } while (0)
                    if (plain) ZG_WALK_ROWS(true); else ZG_WALK_ROWS(false);
#undef ZG_WALK_ROWS
#undef ZG_WALK
                    if (t + n < T) ZG_SEQ_CHECK();
                }
            } else ZG_SEQ_WDT(s.n[9], {
                if (!zg_smem_limit<k_delta_rule<WT>>(((size_t)3 * kDeltaTile * kWalkMaxDim + kDeltaTile) * sizeof(float))) return false;
                launch_pdl(k_delta_rule<WT>, dim3(grid), dim3(kDeltaThreads), smem, st, dst, bufs[s.buf[1]], betab, bufs[s.buf[3]] + s.n[13], wptr<WT>(bufs, s.buf[5], 0), bufs[s.buf[6]],
                                                                  bufs[s.buf[7]], T, H, G, dim, vdim, RS, s.off[0], s.off[1], s.off[2], s.off[3], s.off[4], s.off[5],
                                                                  s.n[5], s.n[6], s.n[7], s.f[1], s.f[2], form, inv_tau, dst_rs, s.n[14]);
            });
            ZG_SEQ_CHECK();
            ZG_SEQ_WDT(s.n[9], launch_pdl(k_delta_out<WT>, dim3((T * H + 3) / 4), dim3(128), 0, st, dst, bufs[s.buf[4]] + s.off[7], wptr<WT>(bufs, s.buf[5], 0), T * H, H, vdim, s.n[8], s.off[6], s.f[0],
                                                           dst_rs, (uint32_t)((form & kDeltaSiluGate) != 0), out_scale, (uint32_t)((form & kDeltaWideNorm) != 0)));
            ZG_SEQ_CHECK();
            return true;
        }
        case ZG_OP_ROUTE: {
            const uint32_t T = s.n[0], NE = s.n[1];
            const uint32_t groups = s.n[5] >= 2 && s.n[6] > 1 ? s.n[6] : 0;
            ZG_SEQ_WDT(s.n[4], launch_pdl(k_route<WT>, dim3((T + 3) / 4), dim3(128), 4 * (NE + groups) * sizeof(float), st, bufs[s.buf[0]], bufs[s.buf[1]] + s.off[1], wptr<WT>(bufs, s.buf[2], s.off[0]), T, NE,
                                                                                         s.n[2], s.n[3], s.n[5], groups, s.n[7], s.f[0]));
            ZG_SEQ_CHECK();
            return true;
        }
        case ZG_OP_MOE_FFN: {
            const uint32_t T = s.n[0], D = s.n[1], ff = s.n[2], E = s.n[3], top = s.n[4];
            if (moe_grouped(s, bufs)) {
                const MoeLayout L = moe_layout(T, D, ff, E, top);
                float* sc = bufs[s.buf[4]];
                const uint32_t run = moe_run(L, ff, zg_sm_count()), segments = L.experts + L.R / run, likely = std::max(L.experts, L.R / run + L.experts / 2);
                ZgExpertSegment* seg = reinterpret_cast<ZgExpertSegment*>(sc + L.seg);
                int* row_pair = reinterpret_cast<int*>(sc + L.row_pair);
                int* pos_of_pair = reinterpret_cast<int*>(sc + L.pos_of_pair);
                launch_pdl(k_moe_sort, dim3(1), dim3(1024), 0, st, bufs[s.buf[2]], seg, row_pair, pos_of_pair, L.R, E, segments, run);
                ZG_SEQ_CHECK();
                launch_pdl(k_moe_gather, dim3(L.R), dim3(256), 0, st, reinterpret_cast<uint32_t*>(sc + L.xs), bufs[s.buf[1]], row_pair, D, top);
                ZG_SEQ_CHECK();
                if (!zg_expert_gemm_launch(wptr<bf16>(bufs, s.buf[3], s.off[0]), wptr<bf16>(bufs, s.buf[3], s.off[1]), E, sc + L.xs, L.R, seg, segments, likely, sc + L.yb, ff, D, s.f[0], s.f[1], s.f[2], st) ||
                    !zg_expert_gemm_launch(wptr<bf16>(bufs, s.buf[3], s.off[2]), nullptr, E, sc + L.yb, L.R, seg, segments, likely, sc + L.z, D, ff, 0.0f, 0.0f, 0.0f, st)) return false;
                launch_pdl(k_moe_combine, dim3(T), dim3(256), 0, st, bufs[s.buf[0]], bufs[s.buf[1]], sc + L.z, bufs[s.buf[2]], pos_of_pair, D, top);
                ZG_SEQ_CHECK();
                return true;
            }
            ZG_SEQ_WDT(s.n[5], {
                if (E && ff) {
                    const uint32_t stage = (size_t)D * 4 <= 48 * 1024 ? 1u : 0u;
                    launch_pdl(k_moe_up<WT>, dim3(dim3((ff + 7) / 8, T * top)), dim3(256), stage ? D * sizeof(float) : 0, st, bufs[s.buf[4]], bufs[s.buf[1]], bufs[s.buf[2]], wptr<WT>(bufs, s.buf[3], s.off[0]),
                                                                           wptr<WT>(bufs, s.buf[3], s.off[1]), D, ff, E, top, s.f[0], s.f[1], s.f[2], stage);
                    ZG_COUNT_LAUNCH();
                }
                launch_pdl(k_moe_down<WT>, dim3(dim3((D + 7) / 8, T)), dim3(256), 0, st, bufs[s.buf[0]], bufs[s.buf[1]], bufs[s.buf[4]], bufs[s.buf[2]], wptr<WT>(bufs, s.buf[3], s.off[2]), D, ff, E, top);
            });
            ZG_SEQ_CHECK();
            return true;
        }
        default:
            if (op.tag >= ZG_OP_STREAM_STEP) return zg_launch_stream_op(op, bufs, st, ahead);
            return op.tag >= ZG_OP_SSM_SCAN ? zg_launch_rec_op(op, bufs, scratch, st) : zg_launch_mix_op(op, bufs, scratch, st, ahead);
    }
}
