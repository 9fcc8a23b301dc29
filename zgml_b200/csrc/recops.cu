// Sequence-model DeviceOps ZG_OP_SSM_SCAN .. ZG_OP_RG_LRU (parameter packs in include/zgml_cuda.h): recurrent mixers
// whose decay is a scalar per head (the state-space scan of Mamba-2) or a gate per element (the minimal gated recurrent
// unit), the gated group norm that closes the former, a per-head RMS norm with a position-dependent temperature, and
// stand-alone activations.  Everything here is f32: step sizes, softplus and exponentials, decays, gates, the states and
// their read-outs, norms and positions.
#include "seq_common.cuh"

#include <math.h>

namespace {

// Walks over many tokens (SSM_SCAN, MIN_GRU from kLongWalk tokens on) are launched WITHOUT programmatic early start.  Such a
// kernel has few CTAs (one per SM or fewer) and is bound by the dependent issue of single warps.  Started early, its CTAs are
// placed while the predecessor's last wave still fills the GPU: on the few SMs that have room, several per SM, where they
// stay for the whole walk and share issue slots.  Measured on a 1024-token step of a 4-layer model at width 2048: 3.02 ms with
// the scan started early, 2.36 ms without (the scan alone: 252 us either way as a one-op program).  Single-token steps keep
// the early start: there the launch gap is what counts.
constexpr int kLongWalk = 64;

// ── SSM_SCAN ─────────────────────────────────────────────────────────────────────────────────────────────────────
// Columns of a head's state S [N, P] evolve independently given the token's B, C, decay and step size, so a head is split by
// columns over CTAs.  A thread keeps a block of 16 RQ state rows x 2 columns in registers (RQ = 1 / 2 / 4 for N <= 128 / 256 /
// 512) as PAIRS OF ROWS: a float4 of B or C read from shared memory is two such pairs as it stands, so the update
// S = a S + B (dt x) and the read-out y += S C are packed f32x2 instructions with no repacking, every B and C value serves
// two columns, and most of the read-out sum stays inside the thread.  (One column and 8 rows per thread was bound by
// shared-memory wavefronts; 4 x 4 blocks by instructions per state element: shuffles, selects and register moves.)  The NS
// threads that share two columns sit in adjacent lanes (NS a power of two <= 8); thread s owns the float4s s + NS i (i < 4 RQ)
// of the rows, so the NS lanes read consecutive float4s.  What is left of the read-out sum crosses the NS lanes in a scatter:
// after the first step a lane carries one of the two columns.
// Step sizes and decays of the head (softplus, two exponentials) are evaluated for a span of tokens at once, in parallel,
// before the walk; B, C and the CTA's x columns arrive in tiles of kSsmTile tokens through cp.async, two tiles in flight, so
// the next tile's loads run under this tile's walk; four tokens are walked per trip so that their loads and sums interleave.
// A step of many tokens in a model with few (head, column block) pairs is cut into segments walked side by side (SsmArgs::mode).
// State in memory: [H][column blocks][32 RQ][kSsmThreads], element (i, thread) — each thread's block, fully coalesced; the
// layout is private to the op (zeros mean an empty state in any layout).
constexpr int kSsmThreads = 128, kSsmTile = 16, kSsmSpan = 1024, kSsmMaxN = 512;
__host__ __device__ inline uint32_t ssm_rq(uint32_t N) { return N > 256 ? 4 : (N > 128 ? 2 : 1); }
__host__ __device__ inline uint32_t ssm_slices(uint32_t N) {
    uint32_t ns = 1;
    while (ns * 16 * ssm_rq(N) < N) ns <<= 1;
    return ns;
}
struct SsmArgs {
    float* dst; const float* xbc; const float* dtl; float* state; const float* ctl;
    uint32_t T, H, G, N, P, x_off, b_off, c_off, dt_off, xbc_rs, dt_rs, vec;
    uint32_t constant;     // form: the decay is a constant per head (a table dtl[H]), the step size 1, and there is no D x in the read-out
    // Segments of a long step walked side by side (the recurrence is linear in the state).  mode 0: the whole step from the carried
    // state.  mode 1: segment blockIdx.z from an EMPTY state, no read-out; leaves the state it reaches and the product of its decays.
    // mode 2: segment blockIdx.z from the state it really starts from (segment 0: the carried one), with the read-out; the last
    // segment leaves the carried state.  Between the two, k_ssm_fold turns the reached states into starting states.
    uint32_t mode, seg_len;
    float* seg_state;      // [segments - 1][state elements of one slot]
    float* seg_decay;      // [segments - 1][H]
};
// global -> shared without passing through registers, 4 or 16 bytes; `on` false writes zeros (nothing is read)
__device__ __forceinline__ void ssm_copy4(float* dst, const float* src, bool on) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int n = on ? 4 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void ssm_copy16(float* dst, const float* src, bool on) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int n = on ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
template <typename WT, uint32_t NS, int RQ>
__global__ void __launch_bounds__(kSsmThreads) k_ssm_scan(SsmArgs a, const WT* __restrict__ a_log, const WT* __restrict__ dt_bias, const WT* __restrict__ dskip) {
    asm volatile("griddepcontrol.wait;" ::: "memory");       // the dependent kernel is let in when the walk is over (below)
    constexpr uint32_t CPB = kSsmThreads / NS * 2, NP = NS * 16 * RQ, NI = 4 * RQ;   // columns per CTA, padded state rows, float4s of rows per thread
    extern __shared__ __align__(16) float sm[];
    constexpr uint32_t kStage = kSsmTile * (2 * NP + CPB);               // per stage: B [tile][NP], C [tile][NP], x [tile][CPB]
    float* Dt = sm + 2 * kStage;                                         // step sizes and decays of a span of tokens
    float* Dec = Dt + kSsmSpan;
    const uint32_t tid = threadIdx.x, s = tid % NS, pl = tid / NS;
    const uint32_t h = blockIdx.y, cb = blockIdx.x, g = h / (a.H / a.G);
    const uint32_t p0 = cb * CPB + pl * 2;                               // this thread's first column
    const uint32_t slot = (uint32_t)ctl_word(a.ctl, ZG_CTL_SLOT);
    const uint32_t n_cb = (a.P + CPB - 1) / CPB;
    constexpr size_t kBlock = (size_t)32 * RQ * kSsmThreads;             // state elements of one (head, column block)
    const size_t slot_elems = (size_t)a.H * n_cb * kBlock, my_block = ((size_t)h * n_cb + cb) * kBlock;
    float* st = a.state + slot * slot_elems + my_block;
    const uint32_t seg = a.mode ? blockIdx.z : 0, n_seg = a.mode ? (a.T + a.seg_len - 1) / a.seg_len : 1;
    const uint32_t t_begin = a.mode ? seg * a.seg_len : 0, t_end = a.mode ? min(a.T, t_begin + a.seg_len) : a.T;
    const float* from = a.mode == 2 && seg > 0 ? a.seg_state + (size_t)(seg - 1) * slot_elems + my_block : st;
    float2 S[NI][2][2];                                                  // [float4 of rows][pair of rows in it][column]
#pragma unroll
    for (int i = 0; i < 16 * RQ; i++) {
        S[i / 4][(i / 2) % 2][i % 2].x = a.mode == 1 ? 0.0f : from[(2 * i) * kSsmThreads + tid];
        S[i / 4][(i / 2) % 2][i % 2].y = a.mode == 1 ? 0.0f : from[(2 * i + 1) * kSsmThreads + tid];
    }
    float decay_product = 1.0f;                                          // mode 1, thread 0
    const bool fixed = a.constant != 0;
    const float neg_a = fixed ? 0.0f : -expf(wld(a_log, h)), bias = fixed ? 0.0f : wld(dt_bias, h), dsk = fixed ? 0.0f : wld(dskip, h);
    const float fixed_decay = fixed ? a.dtl[h] : 0.0f;
    const float* bsrc = a.xbc + a.b_off + (size_t)g * a.N;
    const float* csrc = a.xbc + a.c_off + (size_t)g * a.N;
    const float* xsrc = a.xbc + a.x_off + (size_t)h * a.P + (size_t)cb * CPB;
    const uint32_t x_cols = min(CPB, a.P - cb * CPB);
    // which of its two columns the thread ends up with after the scattered reduction, and whether it is the one that writes it
    const bool up = NS >= 2 && (s & (NS / 2)) != 0;
    const bool writer = NS >= 2 ? (s & (NS / 2 - 1)) == 0 : true;

    auto fetch_tile = [&](uint32_t t0, uint32_t stage) {
        float* Bs = sm + stage * kStage;
        float* Cs = Bs + kSsmTile * NP;
        float* Xs = Cs + kSsmTile * NP;
        const uint32_t nt = min((uint32_t)kSsmTile, t_end - t0);
        if (a.vec) {
            for (uint32_t e = tid; e < nt * (NP / 4); e += kSsmThreads) {
                const uint32_t tt = e / (NP / 4), n = 4 * (e % (NP / 4));
                const bool on = n < a.N;
                ssm_copy16(Bs + tt * NP + n, on ? bsrc + (size_t)(t0 + tt) * a.xbc_rs + n : a.xbc, on);
                ssm_copy16(Cs + tt * NP + n, on ? csrc + (size_t)(t0 + tt) * a.xbc_rs + n : a.xbc, on);
            }
            for (uint32_t e = tid; e < nt * (CPB / 4); e += kSsmThreads) {
                const uint32_t tt = e / (CPB / 4), c = 4 * (e % (CPB / 4));
                const bool on = c < x_cols;
                ssm_copy16(Xs + tt * CPB + c, on ? xsrc + (size_t)(t0 + tt) * a.xbc_rs + c : a.xbc, on);
            }
            return;
        }
        for (uint32_t e = tid; e < nt * NP; e += kSsmThreads) {
            const uint32_t tt = e / NP, n = e % NP;
            const bool on = n < a.N;
            ssm_copy4(Bs + e, on ? bsrc + (size_t)(t0 + tt) * a.xbc_rs + n : a.xbc, on);
            ssm_copy4(Cs + e, on ? csrc + (size_t)(t0 + tt) * a.xbc_rs + n : a.xbc, on);
        }
        for (uint32_t e = tid; e < nt * CPB; e += kSsmThreads) {
            const uint32_t tt = e / CPB, c = e % CPB;
            const bool on = c < x_cols;
            ssm_copy4(Xs + e, on ? xsrc + (size_t)(t0 + tt) * a.xbc_rs + c : a.xbc, on);
        }
    };
    for (uint32_t base = t_begin; base < t_end; base += kSsmSpan) {
        const uint32_t span = min((uint32_t)kSsmSpan, t_end - base);
        __syncthreads();                                   // the previous span's readers are done
        fetch_tile(base, 0);
        asm volatile("cp.async.commit_group;" ::: "memory");
        for (uint32_t t = tid; t < span; t += kSsmThreads) {
            if (fixed) { Dt[t] = 1.0f; Dec[t] = fixed_decay; continue; }
            const float dt = softplusf_(a.dtl[(size_t)(base + t) * a.dt_rs + a.dt_off + h] + bias);
            Dt[t] = dt;
            Dec[t] = expf(neg_a * dt);
        }
        for (uint32_t t0 = 0, it = 0; t0 < span; t0 += kSsmTile, it++) {
            const uint32_t stage = it & 1;
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();                               // tile `it` has landed for everyone, and everyone has left tile it - 1
            if (a.mode == 1 && tid == 0)
                for (uint32_t t = t0; t < min(span, t0 + kSsmTile); t++) decay_product *= Dec[t];
            if (t0 + kSsmTile < span) fetch_tile(base + t0 + kSsmTile, stage ^ 1);
            asm volatile("cp.async.commit_group;" ::: "memory");
            const float* Bs = sm + stage * kStage;
            const float* Cs = Bs + kSsmTile * NP;
            const float* Xs = Cs + kSsmTile * NP;
            const uint32_t nt = min((uint32_t)kSsmTile, span - t0);
            constexpr int U = RQ > 1 ? 2 : 4;              // tokens per trip (4: 238 us per 1024-token walk at 64 heads, 2: 252, 1: 267)
            float* out = a.dst + (size_t)(base + t0) * a.H * a.P + (size_t)h * a.P + p0;
            for (uint32_t tt = 0; tt < nt; tt += U) {
                float2 x[U], d2[U], tx[U][2], y[U][2];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const uint32_t tu = min(tt + u, nt - 1);       // a token past the tile's end repeats the last one with decay 1 and step 0: the state stays
                    const bool live = tt + u < nt;
                    x[u] = *reinterpret_cast<const float2*>(Xs + tu * CPB + pl * 2);
                    const float dec = live ? Dec[t0 + tu] : 1.0f, dt = live ? Dt[t0 + tu] : 0.0f;
                    d2[u] = make_float2(dec, dec);
                    tx[u][0] = make_float2(dt * x[u].x, dt * x[u].x);
                    tx[u][1] = make_float2(dt * x[u].y, dt * x[u].y);
                    y[u][0] = y[u][1] = make_float2(0.0f, 0.0f);
                }
#pragma unroll
                for (int i = 0; i < NI; i++) {
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const uint32_t tu = min(tt + u, nt - 1);
                        const float4 b = *reinterpret_cast<const float4*>(Bs + tu * NP + 4 * (s + NS * i));
                        const float4 c = *reinterpret_cast<const float4*>(Cs + tu * NP + 4 * (s + NS * i));
                        const float2 bp[2] = {make_float2(b.x, b.y), make_float2(b.z, b.w)};     // pairs of rows, as they lie in the registers
                        const float2 cp[2] = {make_float2(c.x, c.y), make_float2(c.z, c.w)};
#pragma unroll
                        for (int k = 0; k < 2; k++)
#pragma unroll
                            for (int j = 0; j < 2; j++) {
                                S[i][k][j] = __ffma2_rn(d2[u], S[i][k][j], __fmul2_rn(bp[k], tx[u][j]));
                                y[u][j] = __ffma2_rn(S[i][k][j], cp[k], y[u][j]);
                            }
                    }
                }
                if (a.mode == 1) continue;                 // no read-out on the walk from an empty state
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const float y0 = y[u][0].x + y[u][0].y, y1 = y[u][1].x + y[u][1].y;
                    if (NS >= 2) {
                        float k = (up ? y1 : y0) + __shfl_xor_sync(0xffffffffu, up ? y0 : y1, NS / 2);
#pragma unroll
                        for (uint32_t o = NS / 4; o > 0; o >>= 1) k += __shfl_xor_sync(0xffffffffu, k, o);
                        const uint32_t col = up ? 1u : 0u;
                        if (writer && tt + u < nt && p0 + col < a.P) out[(size_t)(tt + u) * a.H * a.P + col] = fmaf(dsk, up ? x[u].y : x[u].x, k);
                    } else if (tt + u < nt) {
                        if (p0 < a.P) out[(size_t)(tt + u) * a.H * a.P] = fmaf(dsk, x[u].x, y0);
                        if (p0 + 1 < a.P) out[(size_t)(tt + u) * a.H * a.P + 1] = fmaf(dsk, x[u].y, y1);
                    }
                }
            }
        }
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (a.mode == 2 && seg + 1 < n_seg) return;            // only the last segment leaves the carried state
    float* to = a.mode == 1 ? a.seg_state + (size_t)seg * slot_elems + my_block : st;
#pragma unroll
    for (int i = 0; i < 16 * RQ; i++) {
        to[(2 * i) * kSsmThreads + tid] = S[i / 4][(i / 2) % 2][i % 2].x;
        to[(2 * i + 1) * kSsmThreads + tid] = S[i / 4][(i / 2) % 2][i % 2].y;
    }
    if (a.mode == 1 && cb == 0 && tid == 0) a.seg_decay[(size_t)seg * a.H + h] = decay_product;
}
// Starting states of the segments: start[0] is the carried state, start[j] = (product of segment j - 1's decays) start[j - 1] + the
// state segment j - 1 reached from empty.  start[j] replaces reached[j - 1] in place; one thread per state element.
__global__ void k_ssm_fold(float* __restrict__ seg_state, const float* __restrict__ seg_decay, const float* __restrict__ state, const float* __restrict__ ctl,
                           uint32_t H, uint32_t head_elems, uint32_t n_seg) {
    pdl_enter();
    const size_t slot_elems = (size_t)H * head_elems, e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= slot_elems) return;
    const uint32_t h = (uint32_t)(e / head_elems);
    float s = state[(size_t)ctl_word(ctl, ZG_CTL_SLOT) * slot_elems + e];
    for (uint32_t j = 0; j + 1 < n_seg; j++) {
        s = fmaf(seg_decay[(size_t)j * H + h], s, seg_state[(size_t)j * slot_elems + e]);
        seg_state[(size_t)j * slot_elems + e] = s;
    }
}
static size_t ssm_state_elems(uint32_t H, uint32_t N, uint32_t P) {
    const uint32_t CPB = kSsmThreads / ssm_slices(N) * 2;
    return (size_t)H * ((P + CPB - 1) / CPB) * 32 * ssm_rq(N) * kSsmThreads;
}
// Segments a step is cut into: a walk is bound by the dependent issue of its warps (a warp uses about a quarter of its scheduler's
// issue slots), one CTA per (head, column block), so a long step of a model with few of those is cut while the GPU still holds
// no more than about three CTAs per SM — beyond that the second walk of every token costs more than the segments gain
// (measured at 1024 tokens: 32 heads 252 -> 115 us, 64 heads 252 -> 211 us with five segments, 128 heads 308 -> 373 us with
// three).  A segment has at least 64 tokens.  (Steps of kChunkMinTokens tokens whose rows can be copied 16 bytes at a time go by chunks instead.)
static uint32_t ssm_segments(uint32_t T, uint32_t H, uint32_t N, uint32_t P, uint32_t* seg_len) {
    const uint32_t CPB = kSsmThreads / ssm_slices(N) * 2, ctas = H * ((P + CPB - 1) / CPB);
    uint32_t n = 448 / (ctas ? ctas : 1);
    if (n > 8) n = 8;
    if (n > T / 64) n = T / 64;
    if (n < 2) { *seg_len = T; return 1; }
    const uint32_t len = ((T + n - 1) / n + kSsmTile - 1) / kSsmTile * kSsmTile;
    *seg_len = len;
    return (T + len - 1) / len;
}

// ── SSM_SCAN over many tokens: chunks of 64 ──────────────────────────────────────────────────────────────────────
// A walk token by token reads every B and C value from shared memory for two columns only and waits for its own sums (1024 tokens of 64 heads of
// 128 x 64: two walks of segments, 78 and 131 us; by chunks 38 + 16 + 56 us, of which the products' packed instructions are 15 + 25.  165 tokens of
// 4 heads of 64 x 64 and one token after them: 41 -> 25 us).  By chunks of 64 tokens the step is three products with reuse in both directions, all in f32:
//   S_{c+1} = Gamma_c S_c + sum_s B_s (w_s x_s)^T                   w_s: the step size and the chunk's decays after s
//   y_t     = P_t C_t^T S_c + sum_{s <= t} (C_t . B_s) W_st x_s      P_t: the chunk's decays up to t, W_st: the step size of s and the decays after s up to t
// with only products of decays throughout (nothing is divided by one).  C . B is per group, not per head.
//   k_ssm_chunks:  the sum of the first line per (head, chunk), all chunks side by side; beside them C transposed and C . B per (group, chunk).
//   k_ssm_chain:   the first line's recurrence from chunk to chunk, one thread per four state elements.
//   k_ssm_outputs: the second line, every (chunk, head, 64 columns) a CTA of its own: K = N + 64.
// Products: 8 x 4 outputs per thread as packed pairs, three 16-byte shared loads per 32 of them, sums of 16 terms added to the running ones (a chain of
// 192 would lose a digit to rounding).  Shared-memory wavefronts and the packed instructions share the time about evenly; an 8 x 8 tile per thread would
// halve the former but leave too few registers for the sums of 16.
// From kChunkMinTokens tokens on, where rows can be copied 16 bytes at a time; below two chunks' worth the walk has as little to wait for.
constexpr uint32_t kChunk = 64, kChunkMinTokens = 128, kChunkK = 32, kChunkStages = 3;
constexpr size_t kChunkScratch = (size_t)16 << 20;     // f32 slots of states that one pass over the tokens keeps, half of what the L2 holds (longer steps take several passes)
struct ChunkArgs {
    SsmArgs a;
    uint32_t t0, chunks;                              // this pass: tokens from t0 on
    float4* steps;                                    // [H][chunks * 64]: P_t, decay, step size, w_t
    float* skip;                                      // [H]
    float *ct, *cb, *states;                          // [G][chunks][N][64], [G][chunks][64 s][64 t], [chunks][H][N][P]
};
__host__ __device__ inline uint32_t chunk_count(uint32_t T, uint32_t H, uint32_t N, uint32_t P) {     // per pass
    const size_t fit = kChunkScratch / ((size_t)H * N * P);
    const uint32_t all = (T + kChunk - 1) / kChunk, most = fit < 4 ? 4 : (fit > all ? all : (uint32_t)fit), passes = (all + most - 1) / most;
    return (all + passes - 1) / passes;
}
static size_t chunk_scratch_elems(uint32_t T, uint32_t H, uint32_t G, uint32_t N, uint32_t P) {
    const size_t c = chunk_count(T, H, N, P);
    return (size_t)H * c * kChunk * 4 + (H + 3) / 4 * 4 + (size_t)G * c * (N + kChunk) * kChunk + c * H * N * P;
}
// element of a head's state in the layout of k_ssm_scan
__device__ __forceinline__ size_t ssm_state_at(uint32_t h, uint32_t n, uint32_t p, uint32_t N, uint32_t P, uint32_t NS) {
    const uint32_t RQ = ssm_rq(N), CPB = kSsmThreads / NS * 2, n_cb = (P + CPB - 1) / CPB, i = 4 * (n / 4 / NS) + 2 * ((n / 2) % 2) + p % 2;
    return (((size_t)h * n_cb + p / CPB) * 32 * RQ + 2 * i + n % 2) * kSsmThreads + p % CPB / 2 * NS + (n / 4) % NS;
}
// acc[pair of rows][column] += rows x columns of 16 k; A [k][LDA] at the thread's first row (its other four lie HALF further), B [k][LDB] at its first column.
// FIRST 2: the other four only.
template <uint32_t LDA, uint32_t HALF, uint32_t LDB, int FIRST = 0>
__device__ __forceinline__ void chunk_mma16(float2 (&acc)[4][4], const float* A, const float* B) {
    float2 t[4][4];
#pragma unroll
    for (int k = 0; k < 16; k++) {
        float2 av[4];
#pragma unroll
        for (int i = FIRST; i < 4; i += 2) {
            const float4 x = *reinterpret_cast<const float4*>(A + k * LDA + (i / 2) * HALF);
            av[i] = make_float2(x.x, x.y); av[i + 1] = make_float2(x.z, x.w);
        }
        const float4 b = *reinterpret_cast<const float4*>(B + k * LDB);
        const float bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = FIRST; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float2 bb = make_float2(bv[j], bv[j]);
                t[i][j] = k ? __ffma2_rn(av[i], bb, t[i][j]) : __fmul2_rn(av[i], bb);
            }
    }
#pragma unroll
    for (int i = FIRST; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = __fadd2_rn(acc[i][j], t[i][j]);
}
// a thread's place among TR x TC (of its 128 threads): a warp covers 4 x 8, so that its loads of either operand are few distinct, adjacent float4s
template <uint32_t TR>
__device__ __forceinline__ void chunk_place(uint32_t& tr, uint32_t& tc) {
    const uint32_t warp = (threadIdx.x >> 5) % 4, lane = threadIdx.x & 31;
    tr = warp % (TR / 4) * 4 + lane / 8;
    tc = warp / (TR / 4) * 8 + lane % 8;
}
// A CTA of 256 threads: its halves take every other 16 k; the sums of the second join those of the first (buf: 4096 floats that nobody reads any more).
__device__ __forceinline__ void chunk_join(float2 (&acc)[4][4], float* buf) {
    float4* to = reinterpret_cast<float4*>(buf) + threadIdx.x % 128;
    __syncthreads();
    if (threadIdx.x >= 128)
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j += 2) to[(2 * i + j / 2) * 128] = make_float4(acc[i][j].x, acc[i][j].y, acc[i][j + 1].x, acc[i][j + 1].y);
    __syncthreads();
    if (threadIdx.x < 128)
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j += 2) {
                const float4 x = to[(2 * i + j / 2) * 128];
                acc[i][j] = make_float2(acc[i][j].x + x.x, acc[i][j].y + x.y);
                acc[i][j + 1] = make_float2(acc[i][j + 1].x + x.z, acc[i][j + 1].y + x.w);
            }
}
// decays and step sizes of a head over a chunk, two tokens per lane: (P_t, decay, step size, w_t)
template <typename WT>
__device__ __forceinline__ void chunk_steps(const ChunkArgs& q, uint32_t h, uint32_t c, const WT* a_log, const WT* dt_bias, float4 (&to)[2]) {
    const SsmArgs& a = q.a;
    const uint32_t lane = threadIdx.x & 31;
    const bool fixed = a.constant != 0;
    const float neg_a = fixed ? 0.0f : -expf(wld(a_log, h)), bias = fixed ? 0.0f : wld(dt_bias, h);
    float dt[2], d[2];
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const uint32_t t = q.t0 + c * kChunk + 2 * lane + j;
        dt[j] = t >= a.T ? 0.0f : fixed ? 1.0f : softplusf_(a.dtl[(size_t)t * a.dt_rs + a.dt_off + h] + bias);
        d[j] = t >= a.T ? 1.0f : fixed ? a.dtl[h] : expf(neg_a * dt[j]);
    }
    // in 64 bits, rounded once: equal decays would all round the same way, and 64 of those in a row were 1e-6
    double up = (double)d[0] * d[1], down = up;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double u = __shfl_up_sync(0xffffffffu, up, o), v = __shfl_down_sync(0xffffffffu, down, o);
        if (lane >= (uint32_t)o) up *= u;
        if (lane + o < 32) down *= v;
    }
    double before = __shfl_up_sync(0xffffffffu, up, 1), after = __shfl_down_sync(0xffffffffu, down, 1);
    if (lane == 0) before = 1.0;
    if (lane == 31) after = 1.0;
    to[0] = make_float4((float)(before * d[0]), d[0], dt[0], (float)(after * d[1] * dt[0]));
    to[1] = make_float4((float)up, d[1], dt[1], (float)(after * dt[1]));
}
constexpr uint32_t kProductK = 128, kProductPitch = kProductK + 4;       // n at a time
template <uint32_t NT> constexpr uint32_t chunk_smem() {
    const uint32_t products = (kChunk + 8) * kProductPitch, states = kChunk * (NT + 4096 / NT + 1);      // (at least the 4096 floats of chunk_join)
    return (products > states ? products : states) * (uint32_t)sizeof(float);
}
// First 8 CTAs per (group, chunk): C transposed and C . B, 8 tokens t each.  Then per (head, chunk) and tile of NT state rows x 4096 / NT columns: the state
// that the chunk reaches from an empty one; the first tile leaves the chunk's decays and step sizes.
template <typename WT, uint32_t NT, uint32_t HALVES>
__global__ void __launch_bounds__(128 * HALVES, 4 / HALVES) k_ssm_chunks(ChunkArgs q, const WT* __restrict__ a_log, const WT* __restrict__ dt_bias, const WT* __restrict__ dskip, uint32_t n_tiles, uint32_t p_tiles) {
    pdl_enter();
    constexpr uint32_t kThreads = 128 * HALVES;
    extern __shared__ __align__(16) float sm[];
    const SsmArgs& a = q.a;
    const uint32_t tid = threadIdx.x, products = a.G * q.chunks * 8;
    if (blockIdx.x < products) {
        float* Bs = sm;
        float* Cs = sm + kChunk * kProductPitch;
        const uint32_t part = blockIdx.x % 8, gc = blockIdx.x / 8, g = gc / q.chunks, c = gc % q.chunks, t0 = q.t0 + c * kChunk;
        const uint32_t s = tid % kChunk, tq = tid / kChunk;
        constexpr int kPer = 4 / HALVES;               // tokens t per thread
        // Sums of 16 in f32, those in 64 bits: every output reads these products, and as four f32 chains of 32 terms they made up most of the form's error
        // (1024 tokens of 64 heads of 128 x 64: 1.05e-7 against 64 bits, the walk token by token 9.5e-8 on average over six inputs; now 9.2e-8).
        double total[kPer];
#pragma unroll
        for (int j = 0; j < kPer; j++) total[j] = 0.0;
        for (uint32_t n0 = 0; n0 < a.N; n0 += kProductK) {
            __syncthreads();
#pragma unroll 6
            for (uint32_t e = tid; e < (kChunk + 8) * (kProductK / 4); e += kThreads) {
                const uint32_t r = e / (kProductK / 4), n = 4 * (e % (kProductK / 4)), t = t0 + (r < kChunk ? r : part * 8 + r - kChunk);
                const bool on = t < a.T && n0 + n < a.N;
                ssm_copy16(Bs + r * kProductPitch + n, on ? a.xbc + (size_t)t * a.xbc_rs + (r < kChunk ? a.b_off : a.c_off) + (size_t)g * a.N + n0 + n : a.xbc, on);
            }
            asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
            __syncthreads();
            if (tid < kProductK && n0 + tid < a.N) {
                float* to = q.ct + ((size_t)gc * a.N + n0 + tid) * kChunk + part * 8;
#pragma unroll
                for (int j = 0; j < 8; j += 4)
                    *reinterpret_cast<float4*>(to + j) = make_float4(Cs[j * kProductPitch + tid], Cs[(j + 1) * kProductPitch + tid], Cs[(j + 2) * kProductPitch + tid], Cs[(j + 3) * kProductPitch + tid]);
            }
#pragma unroll 2
            for (uint32_t n16 = 0; n16 < kProductK; n16 += 16) {
                float4 acc[kPer];
#pragma unroll
                for (int j = 0; j < kPer; j++) acc[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
                for (uint32_t n = n16; n < n16 + 16; n += 4) {
                    const float4 b = *reinterpret_cast<const float4*>(Bs + s * kProductPitch + n);
#pragma unroll
                    for (int j = 0; j < kPer; j++) {
                        const float4 x = *reinterpret_cast<const float4*>(Cs + (kPer * tq + j) * kProductPitch + n);
                        acc[j] = make_float4(fmaf(b.x, x.x, acc[j].x), fmaf(b.y, x.y, acc[j].y), fmaf(b.z, x.z, acc[j].z), fmaf(b.w, x.w, acc[j].w));
                    }
                }
#pragma unroll
                for (int j = 0; j < kPer; j++) total[j] += (double)((acc[j].x + acc[j].y) + (acc[j].z + acc[j].w));
            }
        }
#pragma unroll
        for (int j = 0; j < kPer; j += 2)
            *reinterpret_cast<float2*>(q.cb + ((size_t)gc * kChunk + s) * kChunk + part * 8 + kPer * tq + j) =
                make_float2((float)total[j], (float)total[j + 1]);
        return;
    }
    constexpr uint32_t PT = 4096 / NT;
    uint32_t item = blockIdx.x - products;
    const uint32_t nt = item % n_tiles; item /= n_tiles;
    const uint32_t pt = item % p_tiles; item /= p_tiles;
    const uint32_t h = item % a.H, c = item / a.H, g = h / (a.H / a.G), n0 = nt * NT, p0 = pt * PT, t0 = q.t0 + c * kChunk;
    float* Bs = sm;
    float* Xs = Bs + kChunk * NT;
    float* Ws = Xs + kChunk * PT;
#pragma unroll 8
    for (uint32_t e = tid; e < kChunk * NT / 4; e += kThreads) {
        const uint32_t tt = e / (NT / 4), col = n0 + 4 * (e % (NT / 4));
        const bool on = t0 + tt < a.T && col < a.N;
        ssm_copy16(Bs + 4 * e, on ? a.xbc + (size_t)(t0 + tt) * a.xbc_rs + a.b_off + (size_t)g * a.N + col : a.xbc, on);
    }
#pragma unroll 8
    for (uint32_t e = tid; e < kChunk * PT / 4; e += kThreads) {
        const uint32_t tt = e / (PT / 4), col = p0 + 4 * (e % (PT / 4));
        const bool on = t0 + tt < a.T && col < a.P;
        ssm_copy16(Xs + 4 * e, on ? a.xbc + (size_t)(t0 + tt) * a.xbc_rs + a.x_off + (size_t)h * a.P + col : a.xbc, on);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (tid < 32) {
        float4 st[2];
        chunk_steps(q, h, c, a_log, dt_bias, st);
        Ws[2 * tid] = st[0].w;
        Ws[2 * tid + 1] = st[1].w;
        if (nt == 0 && pt == 0) {
            float4* to = q.steps + ((size_t)h * q.chunks + c) * kChunk + 2 * tid;
            to[0] = st[0];
            to[1] = st[1];
            if (c == 0 && tid == 0) q.skip[h] = a.constant ? 0.0f : wld(dskip, h);
        }
    }
    uint32_t tr, tc;
    chunk_place<NT / 8>(tr, tc);
    float2 S[4][4];                                    // [pair of rows][column]
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) S[i][j] = make_float2(0.0f, 0.0f);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (uint32_t e = tid; e < kChunk * PT / 4; e += kThreads) {
        const float w = Ws[e / (PT / 4)];
        float4& x = reinterpret_cast<float4*>(Xs)[e];
        x = make_float4(x.x * w, x.y * w, x.z * w, x.w * w);
    }
    __syncthreads();
    const uint32_t half = tid / 128;
    if (p0 + 32 * (tc / 8) < a.P)                      // uniform over the warp
#pragma unroll 1
        for (uint32_t k = 16 * half; k < kChunk; k += 16 * HALVES) chunk_mma16<NT, NT / 2, PT>(S, Bs + k * NT + 4 * tr, Xs + k * PT + 4 * tc);
    if (HALVES == 2) {
        chunk_join(S, Bs);
        if (half) return;
    }
    const uint32_t p = p0 + 4 * tc;
    float* to = q.states + ((size_t)c * a.H + h) * a.N * a.P + p;
#pragma unroll
    for (int r = 0; r < 8; r++) {
        const uint32_t n = n0 + (r / 4) * (NT / 2) + 4 * tr + r % 4;
        if (n < a.N && p < a.P)
            *reinterpret_cast<float4*>(to + (size_t)n * a.P) = r % 2 ? make_float4(S[r / 2][0].y, S[r / 2][1].y, S[r / 2][2].y, S[r / 2][3].y)
                                                                      : make_float4(S[r / 2][0].x, S[r / 2][1].x, S[r / 2][2].x, S[r / 2][3].x);
    }
}
// The states the chunks reached from empty ones become the states before them; four columns per thread, eight chunks' loads in flight.
__global__ void __launch_bounds__(128) k_ssm_chain(ChunkArgs q, uint32_t NS) {
    pdl_enter();
    const SsmArgs& a = q.a;
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x, per = (size_t)a.H * a.N * a.P;
    if (4 * e >= per) return;
    const uint32_t p = (uint32_t)(4 * e % a.P), n = (uint32_t)(4 * e / a.P % a.N), h = (uint32_t)(4 * e / a.P / a.N), n_cb = (a.P + kSsmThreads / NS * 2 - 1) / (kSsmThreads / NS * 2);
    float* state = a.state + (size_t)ctl_word(a.ctl, ZG_CTL_SLOT) * a.H * n_cb * 32 * ssm_rq(a.N) * kSsmThreads;
    size_t at[4];
    float s[4];
#pragma unroll
    for (int j = 0; j < 4; j++) { at[j] = ssm_state_at(h, n, p + j, a.N, a.P, NS); s[j] = state[at[j]]; }
    float4* z = reinterpret_cast<float4*>(q.states) + e;
    const float4* steps = q.steps + (size_t)h * q.chunks * kChunk;
    for (uint32_t c0 = 0; c0 < q.chunks; c0 += 8) {
        float4 v[8];
        float gamma[8];
#pragma unroll
        for (int i = 0; i < 8; i++)
            if (c0 + i < q.chunks) { v[i] = z[(c0 + i) * (per / 4)]; gamma[i] = steps[(c0 + i + 1) * kChunk - 1].x; }
#pragma unroll
        for (int i = 0; i < 8; i++)
            if (c0 + i < q.chunks) {
                z[(c0 + i) * (per / 4)] = make_float4(s[0], s[1], s[2], s[3]);
                s[0] = fmaf(gamma[i], s[0], v[i].x); s[1] = fmaf(gamma[i], s[1], v[i].y); s[2] = fmaf(gamma[i], s[2], v[i].z); s[3] = fmaf(gamma[i], s[3], v[i].w);
            }
    }
#pragma unroll
    for (int j = 0; j < 4; j++) state[at[j]] = s[j];
}
constexpr uint32_t kChunkOutSmem = (kChunkStages * 2 * kChunkK * kChunk + 5 * kChunk) * sizeof(float);
template <uint32_t HALVES>
__global__ void __launch_bounds__(128 * HALVES, 4 / HALVES) k_ssm_outputs(ChunkArgs q) {
    constexpr uint32_t kThreads = 128 * HALVES;
    pdl_enter();
    extern __shared__ __align__(16) float sm[];
    const SsmArgs& a = q.a;
    constexpr uint32_t stage_elems = 2 * kChunkK * kChunk, PT = 64;
    float4* step = reinterpret_cast<float4*>(sm + kChunkStages * stage_elems);        // [64]
    float* head = reinterpret_cast<float*>(step + kChunk);                             // [64]: decays from the start of the token's 16 up to it
    const uint32_t tid = threadIdx.x, c = blockIdx.x, h = blockIdx.y, g = h / (a.H / a.G), p0 = blockIdx.z * PT;
    uint32_t tr, tc;                                    // rows 4 tr .. + 3 and 32 more, columns 4 tc .. + 3
    chunk_place<8>(tr, tc);
    const uint32_t p = p0 + 4 * tc, half = tid / 128;
    const uint32_t t0 = q.t0 + c * kChunk, n_n = (a.N + kChunkK - 1) / kChunkK, n_stage = n_n + kChunk / kChunkK;
    const float* ct = q.ct + ((size_t)g * q.chunks + c) * a.N * kChunk;
    const float* cb = q.cb + ((size_t)g * q.chunks + c) * kChunk * kChunk;
    const float* st = q.states + ((size_t)c * a.H + h) * a.N * a.P;
    auto fetch = [&](uint32_t i) {
        float* As = sm + i % kChunkStages * stage_elems;
        float* Bs = As + kChunkK * kChunk;
#pragma unroll
        for (uint32_t e = tid; e < kChunkK * kChunk / 4; e += kThreads) {
            const uint32_t r = e / (kChunk / 4), col = p0 + 4 * (e % (kChunk / 4));
            if (i < n_n) {
                const uint32_t n = i * kChunkK + r;
                ssm_copy16(As + 4 * e, n < a.N ? ct + (size_t)i * kChunkK * kChunk + 4 * e : ct, n < a.N);
                const bool on = n < a.N && col < a.P;
                ssm_copy16(Bs + 4 * e, on ? st + (size_t)n * a.P + col : st, on);
            } else {
                const uint32_t s = (i - n_n) * kChunkK + r;
                ssm_copy16(As + 4 * e, cb + (size_t)(i - n_n) * kChunkK * kChunk + 4 * e, true);
                const bool on = t0 + s < a.T && col < a.P;
                ssm_copy16(Bs + 4 * e, on ? a.xbc + (size_t)(t0 + s) * a.xbc_rs + a.x_off + (size_t)h * a.P + col : a.xbc, on);
            }
        }
    };
#pragma unroll
    for (uint32_t i = 0; i < kChunkStages - 1; i++) {
        fetch(i);                                      // n_stage is at least 3
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    const float4* steps = q.steps + ((size_t)h * q.chunks + c) * kChunk;
    if (tid < kChunk) {
        step[tid] = steps[tid];
        double r = 1.0;
        for (uint32_t s = tid / 16 * 16; s <= tid; s++) r *= steps[s].y;
        head[tid] = (float)r;
    }
    float2 acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = make_float2(0.0f, 0.0f);
    for (uint32_t i = 0; i < n_stage; i++) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        if (i + kChunkStages - 1 < n_stage) fetch(i + kChunkStages - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        float* As = sm + i % kChunkStages * stage_elems;
        const float* Bs = As + kChunkK * kChunk;
        bool skip = false;
        if (i >= n_n) {
            if (i == n_n) {                            // the products with the state are complete
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const uint32_t t = (r / 2) * 32 + 4 * tr + 2 * (r % 2);
                    const float2 f = make_float2(step[t].x, step[t + 1].x);
#pragma unroll
                    for (int j = 0; j < 4; j++) acc[r][j] = __fmul2_rn(acc[r][j], f);
                }
            }
            // C . B times W, in place: a thread takes one t and 16 (8) s, from its last to its first
            constexpr uint32_t kRun = 16 / HALVES;
            const uint32_t t = tid % kChunk, s0 = 32 * (i - n_n) + kRun * (tid / kChunk), bs = s0 / 16, bt = t / 16;       // s0 .. + kRun - 1, all of one 16
            float r = 1.0f;
            if (bs < bt) {
                r = head[t];
                for (uint32_t b = bs + 1; b < bt; b++) r *= head[16 * b + 15];
            }
            for (uint32_t s = s0 + kRun; s < 16 * bs + 16; s++)
                if (s <= t) r *= step[s].y;
            bool finite = true;
#pragma unroll
            for (int k = kRun - 1; k >= 0; k--) {
                const uint32_t s = s0 + k, at = (s % kChunkK) * kChunk + t;
                const float4 f = step[s];
                const bool seen = s <= t;
                As[at] = seen ? As[at] * (r * f.z) : 0.0f;
                if (seen) r *= f.y;
                finite &= fabsf(Bs[at]) <= 3.4028234e38f;
            }
            skip = __syncthreads_or(!finite);
        }
        if (!skip) {
#pragma unroll 1
            for (uint32_t k = 16 * half; k < kChunkK; k += 16 * HALVES)
                if (i == n_n + 1) chunk_mma16<kChunk, 32, kChunk, 2>(acc, As + k * kChunk + 4 * tr, Bs + k * kChunk + 4 * tc);      // tokens from 32 on: the first 32 rows have not seen them
                else chunk_mma16<kChunk, 32, kChunk>(acc, As + k * kChunk + 4 * tr, Bs + k * kChunk + 4 * tc);
        } else {                                       // an x that is not finite must not meet the zeros of earlier tokens
#pragma unroll 1
            for (uint32_t kk = 16 * half; kk < kChunkK; kk += kk % 16 == 15 ? 16 * HALVES - 15 : 1) {
                const uint32_t s = (i - n_n) * kChunkK + kk;
                for (uint32_t r = 0; r < 8; r++)
                    for (uint32_t j = 0; j < 4; j++) {
                        const uint32_t row = (r / 4) * 32 + 4 * tr + r % 4;
                        const float v = As[kk * kChunk + row] * Bs[kk * kChunk + 4 * tc + j];
#pragma unroll
                        for (uint32_t rr = 0; rr < 4; rr++)
#pragma unroll
                            for (uint32_t jj = 0; jj < 4; jj++)
                                if (r / 2 == rr && j == jj && s <= row) { if (r % 2) acc[rr][jj].y += v; else acc[rr][jj].x += v; }
                    }
            }
        }
    }
    if (HALVES == 2) {
        chunk_join(acc, sm);
        if (half) return;
    }
    const float dsk = q.skip[h];
#pragma unroll
    for (int r = 0; r < 8; r++) {
        const uint32_t t = t0 + (r / 4) * 32 + 4 * tr + r % 4;
        if (t >= a.T || p >= a.P) continue;
        const float4 x = *reinterpret_cast<const float4*>(a.xbc + (size_t)t * a.xbc_rs + a.x_off + (size_t)h * a.P + p);
        const float y[4] = {r % 2 ? acc[r / 2][0].y : acc[r / 2][0].x, r % 2 ? acc[r / 2][1].y : acc[r / 2][1].x, r % 2 ? acc[r / 2][2].y : acc[r / 2][2].x, r % 2 ? acc[r / 2][3].y : acc[r / 2][3].x};
        *reinterpret_cast<float4*>(a.dst + ((size_t)t * a.H + h) * a.P + p) = make_float4(fmaf(dsk, x.x, y[0]), fmaf(dsk, x.y, y[1]), fmaf(dsk, x.z, y[2]), fmaf(dsk, x.w, y[3]));
    }
}

// ── MIN_GRU, RG_LRU: gated recurrences per channel ───────────────────────────────────────────────────────────────
// S_t = a_t S_{t-1} + b_t is a linear recurrence per channel whose coefficients do not depend on the state, so the step's
// tokens are cut into up to 64 segments that are walked side by side: thread (channel, segment) first walks its segment
// from an empty state, keeping the product of the a_t and the value reached; the segments' (product, value) pairs are then
// folded in order, which gives every segment the state it starts from; the second walk writes the outputs.  A single-token
// step is one segment of one token.  A CELL names the recurrence: what it reads per (token, channel), what it keeps per
// channel, how a token advances (product, state), and what leaves the unit.
constexpr int kGruChannels = 16, kGruMaxSegments = 64;
// minimal gated recurrent unit: z = sigmoid(zl), candidate u + 1/2 (u >= 0) or sigmoid(u), S <- (1 - z) S + z c, out = S silu(g)
struct MinGruCell {
    const float* proj; uint32_t rs, z_off, u_off, g_off;
    struct Chan {};
    struct Raw { float zl, u, gl; };
    __device__ __forceinline__ Chan channel(uint32_t) const { return Chan(); }
    __device__ __forceinline__ Raw load(uint32_t t, uint32_t c, bool out) const {
        const float* row = proj + (size_t)t * rs;
        Raw r; r.zl = row[z_off + c]; r.u = row[u_off + c]; r.gl = out ? row[g_off + c] : 0.0f;
        return r;
    }
    __device__ __forceinline__ void step(const Chan&, const Raw& r, float& A, float& S) const {
        const float z = sigmoidf_(r.zl), cand = r.u >= 0.0f ? r.u + 0.5f : sigmoidf_(r.u);
        A *= 1.0f - z;
        S = fmaf(z, cand, (1.0f - z) * S);
    }
    __device__ __forceinline__ float out(const Raw& r, float S) const { return S * (r.gl * sigmoidf_(r.gl)); }
};
// real-gated linear recurrent unit: r = sigmoid(rl + br), i = sigmoid(il + bi), log a = -c r softplus(lam),
// S <- a S + sqrt(1 - a^2) (i u), out = S act(y).  1 - a^2 = -expm1(2 log a) keeps its digits where a is close to 1.
template <typename WT>
struct RgLruCell {
    const float* u; const float* gates; const float* y; const WT* wts;
    uint32_t u_rs, u_off, g_rs, r_off, i_off, g_bw, g_bs, y_rs, y_off, rb_off, ib_off, lam_off, act;
    float c;
    struct Chan { float br, bi, rate; uint32_t gcol; };
    struct Raw { float rl, il, u, y; };
    __device__ __forceinline__ Chan channel(uint32_t ch) const {
        Chan k; k.br = wld(wts, (size_t)rb_off + ch); k.bi = wld(wts, (size_t)ib_off + ch); k.rate = c * softplusf_(wld(wts, (size_t)lam_off + ch));
        k.gcol = (ch / g_bw) * g_bs + ch % g_bw;
        return k;
    }
    __device__ __forceinline__ Raw load(uint32_t t, uint32_t ch, bool out) const {
        const uint32_t gcol = (ch / g_bw) * g_bs + ch % g_bw;
        const float* g = gates + (size_t)t * g_rs + gcol;
        Raw r; r.rl = g[r_off]; r.il = g[i_off]; r.u = u[(size_t)t * u_rs + u_off + ch]; r.y = out ? y[(size_t)t * y_rs + y_off + ch] : 0.0f;
        return r;
    }
    __device__ __forceinline__ void step(const Chan& k, const Raw& r, float& A, float& S) const {
        const float la = -k.rate * sigmoidf_(r.rl + k.br), a = expf(la);
        A *= a;
        S = fmaf(a, S, sqrtf(-expm1f(2.0f * la)) * (sigmoidf_(r.il + k.bi) * r.u));
    }
    __device__ __forceinline__ float out(const Raw& r, float S) const { return S * seq_epilogue(r.y, act); }
};
template <typename Cell>
__global__ void __launch_bounds__(kGruChannels * kGruMaxSegments) k_channel_scan(Cell cell, float* __restrict__ dst, float* __restrict__ state,
                                                                                 const float* __restrict__ ctl, uint32_t T, uint32_t W, uint32_t drs, uint32_t seg_len) {
    pdl_enter();
    __shared__ float segA[kGruMaxSegments][kGruChannels], segB[kGruMaxSegments][kGruChannels];
    const uint32_t c = blockIdx.x * kGruChannels + threadIdx.x, seg = threadIdx.y, n_seg = blockDim.y;
    const bool on = c < W;
    const uint32_t t_begin = min(T, seg * seg_len), t_end = min(T, t_begin + seg_len);
    float* st = state + (size_t)ctl_word(ctl, ZG_CTL_SLOT) * W;
    const typename Cell::Chan chan = cell.channel(on ? c : 0);
    float S = 0.0f;
    constexpr int U = 8;                                   // tokens whose loads are in flight together
    if (n_seg > 1) {
        float A = 1.0f;
        if (on)
            for (uint32_t t = t_begin; t < t_end; t += U) {
                typename Cell::Raw raw[U];
#pragma unroll
                for (int i = 0; i < U; i++) raw[i] = cell.load(min(t + i, t_end - 1), c, false);
#pragma unroll
                for (int i = 0; i < U; i++)
                    if (t + i < t_end) cell.step(chan, raw[i], A, S);
            }
        segA[seg][threadIdx.x] = A;
        segB[seg][threadIdx.x] = S;
        __syncthreads();
    }
    if (!on) return;
    S = st[c];
    for (uint32_t j = 0; j < seg; j++) S = fmaf(segA[j][threadIdx.x], S, segB[j][threadIdx.x]);
    for (uint32_t t = t_begin; t < t_end; t += U) {
        typename Cell::Raw raw[U];
#pragma unroll
        for (int i = 0; i < U; i++) raw[i] = cell.load(min(t + i, t_end - 1), c, true);
#pragma unroll
        for (int i = 0; i < U; i++) {
            if (t + i < t_end) {
                float A = 1.0f;
                cell.step(chan, raw[i], A, S);
                dst[(size_t)(t + i) * drs + c] = cell.out(raw[i], S);
            }
        }
    }
    if (seg == n_seg - 1) st[c] = S;
}
// segments of a step of T tokens: four tokens or more each, no empty one at the end (the last leaves the state behind)
static uint32_t scan_segments(uint32_t T, uint32_t* seg_len) {
    uint32_t n_seg = (T + 3) / 4;
    if (n_seg > (uint32_t)kGruMaxSegments) n_seg = kGruMaxSegments;
    *seg_len = (T + n_seg - 1) / n_seg;
    return (T + *seg_len - 1) / *seg_len;
}

// ── GATED_NORM: one CTA per (token, group) ───────────────────────────────────────────────────────────────────────
// forms (op parameter n7): the gate multiplies what the norm returns instead of what it reads; a sigmoid gate instead of SiLU
constexpr uint32_t kGateAfter = 1, kGateSigmoid = 2;
__device__ __forceinline__ float gated_norm_gate(float z, uint32_t form) { return (form & kGateSigmoid) ? sigmoidf_(z) : z * sigmoidf_(z); }
template <typename WT>
__global__ void k_gated_norm(float* dst, const float* src, const float* __restrict__ gate, const WT* __restrict__ w, uint32_t cols, uint32_t groups,
                             uint32_t gate_rs, uint32_t src_rs, uint32_t dst_rs, float eps, uint32_t form) {
    pdl_enter();
    __shared__ float sh[32];
    const uint32_t t = blockIdx.x / groups, gi = blockIdx.x % groups, gs = cols / groups, c0 = gi * gs;
    const float* x = src + (size_t)t * src_rs + c0;
    const float* gt = gate + (size_t)t * gate_rs + c0;
    float* out = dst + (size_t)t * dst_rs + c0;
    constexpr int kKeep = 8;                               // values a thread keeps: groups of up to 8 x blockDim are read once, all loads in flight together
    if (gs <= kKeep * blockDim.x) {
        float v[kKeep], z[kKeep], wv[kKeep];
#pragma unroll
        for (int i = 0; i < kKeep; i++) {
            const uint32_t c = threadIdx.x + i * blockDim.x;
            v[i] = c < gs ? x[c] : 0.0f;
            z[i] = c < gs ? gt[c] : 0.0f;
            wv[i] = c < gs ? wld(w, c0 + c) : 0.0f;
        }
        float q = 0.0f;
#pragma unroll
        for (int i = 0; i < kKeep; i++) {
            z[i] = gated_norm_gate(z[i], form);
            if (form & kGateAfter) wv[i] *= z[i]; else v[i] *= z[i];
            q = fmaf(v[i], v[i], q);
        }
        const float inv = 1.0f / sqrtf(block_sum(q, sh) / (float)gs + eps);
#pragma unroll
        for (int i = 0; i < kKeep; i++) {
            const uint32_t c = threadIdx.x + i * blockDim.x;
            if (c < gs) out[c] = v[i] * inv * wv[i];
        }
        return;
    }
    float q = 0.0f;
    for (uint32_t c = threadIdx.x; c < gs; c += blockDim.x) {
        const float v = (form & kGateAfter) ? x[c] : x[c] * gated_norm_gate(gt[c], form);
        q = fmaf(v, v, q);
    }
    const float inv = 1.0f / sqrtf(block_sum(q, sh) / (float)gs + eps);
    for (uint32_t c = threadIdx.x; c < gs; c += blockDim.x) {
        out[c] = x[c] * gated_norm_gate(gt[c], form) * inv * wld(w, c0 + c);
    }
}

// ── HEAD_NORM: one warp per (token, head), in place ──────────────────────────────────────────────────────────────
template <typename WT>
__global__ void k_head_norm(float* x, const WT* __restrict__ w, const float* __restrict__ ctl, uint32_t T, uint32_t heads, uint32_t dim, uint32_t rs,
                            uint32_t period, float eps, float coef) {
    pdl_enter();
    const uint32_t item = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (item >= T * heads) return;
    const uint32_t t = item / heads, hd = item % heads;
    float* v = x + (size_t)t * rs + (size_t)hd * dim;
    float q = 0.0f;
    for (uint32_t c = lane; c < dim; c += 32) q = fmaf(v[c], v[c], q);
    float mult = 1.0f / sqrtf(warp_sum(q) / (float)dim + eps);
    if (period) {
        const uint32_t pos = (uint32_t)ctl_word(ctl, ZG_CTL_POS) + t;
        mult *= fmaf(coef, logf((float)((pos + 1) / period) + 1.0f), 1.0f);
    }
    for (uint32_t c = lane; c < dim; c += 32) v[c] = v[c] * wld(w, c) * mult;
}

// ── ACTIVATION ───────────────────────────────────────────────────────────────────────────────────────────────────
// four elements per thread (n a multiple of 4, both buffers on 16-byte boundaries) or one
template <bool VEC>
__global__ void k_activation(float* dst, const float* src, uint32_t n, uint32_t kind, float p) {
    pdl_enter();
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (VEC) {
        if (4 * e >= n) return;
        float4 v = reinterpret_cast<const float4*>(src)[e];
        v.x = seq_activation(v.x, kind, p); v.y = seq_activation(v.y, kind, p); v.z = seq_activation(v.z, kind, p); v.w = seq_activation(v.w, kind, p);
        reinterpret_cast<float4*>(dst)[e] = v;
    } else {
        if (e >= n) return;
        dst[e] = seq_activation(src[e], kind, p);
    }
}

}  // namespace

// shared scratch of a long SSM_SCAN step: by chunks (whether its rows are aligned for that is known at the launch), or per segment but the last a state
// (reached, then starting) and the product of its decays per head
size_t zg_rec_op_scratch_elems(const ZgOp& op) {
    if (op.tag != ZG_OP_SSM_SCAN) return 0;
    const ZgSeqOp& s = op.u.seq;
    if (!s.n[1] || !s.n[3] || !s.n[4] || s.n[3] > (uint32_t)kSsmMaxN) return 0;
    uint32_t len;
    const uint32_t n = ssm_segments(s.n[0], s.n[1], s.n[3], s.n[4], &len);
    const size_t walks = n > 1 ? (size_t)(n - 1) * (ssm_state_elems(s.n[1], s.n[3], s.n[4]) + s.n[1]) : 0;
    const size_t chunks = s.n[0] >= kChunkMinTokens && s.n[2] ? chunk_scratch_elems(s.n[0], s.n[1], s.n[2], s.n[3], s.n[4]) : 0;
    return walks > chunks ? walks : chunks;
}

// f32 slots per state slot of an op whose state layout is its own (SSM_SCAN); 0 for every other op
extern "C" __attribute__((visibility("default"))) size_t zg_cuda_seq_state_elems(const ZgOp* op) {
    if (!op || op->tag != ZG_OP_SSM_SCAN) return 0;
    const ZgSeqOp& s = op->u.seq;
    if (!s.n[1] || !s.n[3] || !s.n[4] || s.n[3] > (uint32_t)kSsmMaxN) return 0;
    return ssm_state_elems(s.n[1], s.n[3], s.n[4]);
}

bool zg_rec_op_valid(const ZgOp& op, const size_t* elems, size_t n_bufs, char* why, size_t why_n) {
    const ZgSeqOp& s = op.u.seq;
    auto fail = [&](const char* m) { snprintf(why, why_n, "%s", m); return false; };
    auto have = [&](int i) { return s.buf[i] != ZG_NO_BUF && s.buf[i] < n_bufs; };
    auto fits = [&](int i, size_t off, size_t n) { return have(i) && off + n <= elems[s.buf[i]]; };
    auto wfits = [&](int i, uint32_t wdt, size_t off, size_t n) { return wdt <= ZG_W_BF16 && have(i) && (wdt == ZG_W_BF16 ? (off + n + 1) / 2 : off + n) <= elems[s.buf[i]]; };
    switch (op.tag) {
        case ZG_OP_SSM_SCAN: {
            const size_t T = s.n[0], H = s.n[1], G = s.n[2], N = s.n[3], P = s.n[4], xrs = s.n[5], drs = s.n[6];
            if (!T || !H || !G || H % G || !N || N > (size_t)kSsmMaxN || !P) return fail("ssm_scan: shape");
            const bool fixed = s.n[8] != 0;        // constant decays: a table instead of the dt rows, no weights
            if (s.n[8] > 1 || s.off[0] + H * P > xrs || s.off[1] + G * N > xrs || s.off[2] + G * N > xrs || (!fixed && s.off[3] + H > drs)) return fail("ssm_scan: columns");
            if (!fits(0, 0, T * H * P) || !fits(1, 0, T * xrs) || !fits(2, fixed ? s.off[3] : 0, fixed ? H : T * drs) ||
                (!fixed && (!wfits(3, s.n[7], s.off[4], H) || !wfits(3, s.n[7], s.off[5], H) || !wfits(3, s.n[7], s.off[6], H))) || !have(4) || elems[s.buf[4]] < ssm_state_elems((uint32_t)H, (uint32_t)N, (uint32_t)P) || !fits(5, 0, ZG_CTL_IDS))
                return fail("ssm_scan: extent");
            if (s.buf[0] == s.buf[1] || s.buf[0] == s.buf[2]) return fail("ssm_scan: in place");
            return true;
        }
        case ZG_OP_MIN_GRU: {
            const size_t T = s.n[0], W = s.n[1], rs = s.n[2], drs = s.n[3];
            if (!T || !W || drs < W || s.off[0] + W > rs || s.off[1] + W > rs || s.off[2] + W > rs) return fail("min_gru: shape");
            if (!fits(0, 0, (T - 1) * drs + W) || !fits(1, 0, T * rs) || !have(2) || elems[s.buf[2]] < W || !fits(3, 0, ZG_CTL_IDS)) return fail("min_gru: extent");
            if (s.buf[0] == s.buf[1]) return fail("min_gru: in place");
            return true;
        }
        case ZG_OP_GATED_NORM: {
            const size_t T = s.n[0], cols = s.n[1], groups = s.n[2], grs = s.n[3], srs = s.n[5], drs = s.n[6];
            if (!T || !cols || !groups || cols % groups || srs < cols || drs < cols || s.off[0] + cols > grs || s.n[7] > 3) return fail("gated_norm: shape");
            if (!fits(0, 0, (T - 1) * drs + cols) || !fits(1, 0, (T - 1) * srs + cols) || !fits(2, 0, (T - 1) * grs + s.off[0] + cols) || !wfits(3, s.n[4], s.off[1], cols))
                return fail("gated_norm: extent");
            return true;
        }
        case ZG_OP_HEAD_NORM: {
            const size_t T = s.n[0], heads = s.n[1], dim = s.n[2], rs = s.n[3];
            if (!T || !heads || !dim || s.off[0] + heads * dim > rs) return fail("head_norm: shape");
            if (!fits(0, 0, (T - 1) * rs + s.off[0] + heads * dim) || !wfits(1, s.n[4], s.off[1], dim) || !fits(2, 0, ZG_CTL_IDS)) return fail("head_norm: extent");
            return true;
        }
        case ZG_OP_RG_LRU: {
            const size_t T = s.n[0], W = s.n[1], urs = s.n[2], grs = s.n[3], bw = s.n[4], bs = s.n[5], yrs = s.n[6], drs = s.n[7];
            if (!T || !W || !bw || W % bw || bs < bw || drs < W || s.n[9] > 6 || !(s.f[0] > 0.0f)) return fail("rg_lru: shape");
            const size_t gspan = (W / bw - 1) * bs + bw;
            if (s.off[0] + W > urs || s.off[1] + gspan > grs || s.off[2] + gspan > grs || s.off[3] + W > yrs) return fail("rg_lru: columns");
            if (!fits(0, 0, (T - 1) * drs + W) || !fits(1, 0, (T - 1) * urs + s.off[0] + W) || !fits(2, 0, (T - 1) * grs + (s.off[1] > s.off[2] ? s.off[1] : s.off[2]) + gspan) ||
                !fits(3, 0, (T - 1) * yrs + s.off[3] + W) || !wfits(4, s.n[8], s.off[4], W) || !wfits(4, s.n[8], s.off[5], W) || !wfits(4, s.n[8], s.off[6], W) || !have(5) ||
                elems[s.buf[5]] < W || !fits(6, 0, ZG_CTL_IDS))
                return fail("rg_lru: extent");
            if (s.buf[0] == s.buf[1] || s.buf[0] == s.buf[2] || s.buf[0] == s.buf[3]) return fail("rg_lru: in place");
            return true;
        }
        case ZG_OP_ACTIVATION: {
            if (!s.n[0] || s.n[1] > 5 || (s.n[1] == 4 && !(s.f[0] > 0.0f))) return fail("activation: shape");
            if (!fits(0, 0, s.n[0]) || !fits(1, 0, s.n[0])) return fail("activation: extent");
            return true;
        }
        default: return fail("not a sequence op");
    }
}

uint32_t zg_rec_op_writes(uint32_t tag) {
    switch (tag) {
        case ZG_OP_SSM_SCAN: return 1u | (1u << 4);
        case ZG_OP_MIN_GRU: return 1u | (1u << 2);
        case ZG_OP_RG_LRU: return 1u | (1u << 5);
        default: return 1u;
    }
}

bool zg_launch_rec_op(const ZgOp& op, float* const* bufs, float* scratch, cudaStream_t st) {
    const ZgSeqOp& s = op.u.seq;
    switch (op.tag) {
        case ZG_OP_SSM_SCAN: {
            SsmArgs a;
            a.dst = bufs[s.buf[0]]; a.xbc = bufs[s.buf[1]]; a.dtl = bufs[s.buf[2]]; a.state = bufs[s.buf[4]]; a.ctl = bufs[s.buf[5]];
            a.T = s.n[0]; a.H = s.n[1]; a.G = s.n[2]; a.N = s.n[3]; a.P = s.n[4]; a.x_off = s.off[0]; a.b_off = s.off[1]; a.c_off = s.off[2]; a.dt_off = s.off[3];
            a.xbc_rs = s.n[5]; a.dt_rs = s.n[6]; a.constant = s.n[8];
            if (a.constant) a.dtl += s.off[3];
            const uint32_t NS = ssm_slices(a.N), RQ = ssm_rq(a.N), CPB = kSsmThreads / NS * 2;
            // 16-byte copies when every row of B, C and the CTA's x columns starts on a 16-byte boundary
            a.vec = (a.N % 4 == 0 && a.P % 4 == 0 && a.xbc_rs % 4 == 0 && a.x_off % 4 == 0 && a.b_off % 4 == 0 && a.c_off % 4 == 0 &&
                     (reinterpret_cast<uintptr_t>(a.xbc) & 15) == 0) ? 1u : 0u;
            const size_t smem = ((size_t)2 * kSsmTile * (2 * NS * 16 * RQ + CPB) + 2 * kSsmSpan) * sizeof(float);
            const size_t slot_elems = ssm_state_elems(a.H, a.N, a.P);
            if (scratch && a.T >= kChunkMinTokens && a.vec && (reinterpret_cast<uintptr_t>(a.dst) & 15) == 0) {
                ChunkArgs q;
                q.a = a;
                const uint32_t most = chunk_count(a.T, a.H, a.N, a.P);
                q.steps = reinterpret_cast<float4*>(scratch);
                q.skip = scratch + (size_t)a.H * most * kChunk * 4;
                q.ct = q.skip + (a.H + 3) / 4 * 4;
                q.cb = q.ct + (size_t)a.G * most * a.N * kChunk;
                q.states = q.cb + (size_t)a.G * most * kChunk * kChunk;
                for (q.t0 = 0; q.t0 < a.T; q.t0 += most * kChunk) {
                    const uint32_t left = (a.T - q.t0 + kChunk - 1) / kChunk;
                    q.chunks = left < most ? left : most;
                    const uint32_t NT = a.N <= 32 ? 32 : a.N <= 64 ? 64 : 128, n_tiles = (a.N + NT - 1) / NT, p_tiles = (a.P + 4096 / NT - 1) / (4096 / NT);
                    const dim3 cgrid(a.G * q.chunks * 8 + a.H * q.chunks * n_tiles * p_tiles);
                    // The GPU holds about four CTAs of 128 threads per SM; a grid of fewer than two per SM is bound by the latency of each, and takes
                    // twice the threads for it (224 tokens, 64 heads of 64 x 64: 39 us instead of 45; at 384 CTAs, 349 tokens of 32 heads of 64 x 128,
                    // 47 us with 128 threads and 55 with 256).
                    const dim3 ogrid(q.chunks, a.H, (a.P + 63) / 64);
                    const bool few = ogrid.x * ogrid.y * ogrid.z <= 296;
#define ZG_SSM_CHUNKS(NT_, HALVES_)                                                                                                           \
    ZG_SEQ_WDT(s.n[7], launch_pdl(k_ssm_chunks<WT, NT_, HALVES_>, cgrid, dim3(128 * HALVES_), chunk_smem<NT_>(), st, q, a.constant ? (const WT*)nullptr : (const WT*)wptr<WT>(bufs, s.buf[3], s.off[4]), \
                                  a.constant ? (const WT*)nullptr : (const WT*)wptr<WT>(bufs, s.buf[3], s.off[5]), a.constant ? (const WT*)nullptr : (const WT*)wptr<WT>(bufs, s.buf[3], s.off[6]), n_tiles, p_tiles))
                    if (few) {
                        if (NT == 32) ZG_SSM_CHUNKS(32, 2); else if (NT == 64) ZG_SSM_CHUNKS(64, 2); else ZG_SSM_CHUNKS(128, 2);
                    } else if (NT == 32) ZG_SSM_CHUNKS(32, 1); else if (NT == 64) ZG_SSM_CHUNKS(64, 1); else ZG_SSM_CHUNKS(128, 1);
#undef ZG_SSM_CHUNKS
                    ZG_SEQ_CHECK();
                    launch_pdl(k_ssm_chain, dim3((unsigned)(((size_t)a.H * a.N * a.P / 4 + 127) / 128)), dim3(128), 0, st, q, NS);
                    ZG_SEQ_CHECK();
                    if (few) {
                        cudaFuncSetAttribute(k_ssm_outputs<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kChunkOutSmem);
                        launch_pdl(k_ssm_outputs<2>, ogrid, dim3(256), kChunkOutSmem, st, q);
                    } else {
                        cudaFuncSetAttribute(k_ssm_outputs<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kChunkOutSmem);
                        launch_pdl(k_ssm_outputs<1>, ogrid, dim3(128), kChunkOutSmem, st, q);
                    }
                    ZG_SEQ_CHECK();
                }
                return true;
            }
            uint32_t seg_len = a.T;
            const uint32_t n_seg = scratch ? ssm_segments(a.T, a.H, a.N, a.P, &seg_len) : 1;
            a.seg_len = seg_len;
            a.seg_state = scratch;
            a.seg_decay = scratch ? scratch + (size_t)(n_seg > 1 ? n_seg - 1 : 0) * slot_elems : nullptr;
#define ZG_SSM(NS_, RQ_)                                                                                                                  \
    ZG_SEQ_WDT(s.n[7], {                                                                                                                  \
        if (smem > 48 * 1024) cudaFuncSetAttribute(k_ssm_scan<WT, NS_, RQ_>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);     \
        launch_pdl_if(a.T < (uint32_t)kLongWalk, k_ssm_scan<WT, NS_, RQ_>, grid, dim3(kSsmThreads), smem, st, a, a.constant ? (const WT*)nullptr : (const WT*)wptr<WT>(bufs, s.buf[3], s.off[4]), \
                      a.constant ? (const WT*)nullptr : (const WT*)wptr<WT>(bufs, s.buf[3], s.off[5]), a.constant ? (const WT*)nullptr : (const WT*)wptr<WT>(bufs, s.buf[3], s.off[6]));                                            \
    })
#define ZG_SSM_ANY()                                                                                                                      \
    do {                                                                                                                                  \
        if (RQ == 4) ZG_SSM(8, 4);                                                                                                        \
        else if (RQ == 2) ZG_SSM(8, 2);                                                                                                   \
        else switch (NS) {                                                                                                                \
            case 1: ZG_SSM(1, 1); break;                                                                                                  \
            case 2: ZG_SSM(2, 1); break;                                                                                                  \
            case 4: ZG_SSM(4, 1); break;                                                                                                  \
            default: ZG_SSM(8, 1); break;                                                                                                 \
        }                                                                                                                                 \
    } while (0)
            dim3 grid((a.P + CPB - 1) / CPB, a.H, 1);
            if (n_seg > 1) {       // every segment but the last from an empty state, the fold, then every segment from its real start
                a.mode = 1; grid.z = n_seg - 1;
                ZG_SSM_ANY();
                ZG_SEQ_CHECK();
                launch_pdl(k_ssm_fold, dim3((unsigned)((slot_elems + 255) / 256)), dim3(256), 0, st, a.seg_state, (const float*)a.seg_decay, (const float*)a.state, a.ctl, a.H,
                           (uint32_t)(slot_elems / a.H), n_seg);
                ZG_SEQ_CHECK();
                a.mode = 2; grid.z = n_seg;
                ZG_SSM_ANY();
            } else {
                a.mode = 0;
                ZG_SSM_ANY();
            }
#undef ZG_SSM_ANY
#undef ZG_SSM
            ZG_SEQ_CHECK();
            return true;
        }
        case ZG_OP_MIN_GRU: {
            const uint32_t T = s.n[0];
            uint32_t seg_len;
            const uint32_t n_seg = scan_segments(T, &seg_len);
            MinGruCell cell;
            cell.proj = bufs[s.buf[1]]; cell.rs = s.n[2]; cell.z_off = s.off[0]; cell.u_off = s.off[1]; cell.g_off = s.off[2];
            launch_pdl_if(T < (uint32_t)kLongWalk, k_channel_scan<MinGruCell>, dim3((s.n[1] + kGruChannels - 1) / kGruChannels), dim3(kGruChannels, n_seg), 0, st, cell, bufs[s.buf[0]], bufs[s.buf[2]],
                          (const float*)bufs[s.buf[3]], T, s.n[1], s.n[3], seg_len);
            ZG_SEQ_CHECK();
            return true;
        }
        case ZG_OP_RG_LRU: {
            const uint32_t T = s.n[0];
            uint32_t seg_len;
            const uint32_t n_seg = scan_segments(T, &seg_len);
            ZG_SEQ_WDT(s.n[8], {
                RgLruCell<WT> cell;
                cell.u = bufs[s.buf[1]]; cell.gates = bufs[s.buf[2]]; cell.y = bufs[s.buf[3]]; cell.wts = wptr<WT>(bufs, s.buf[4], 0);
                cell.u_rs = s.n[2]; cell.u_off = s.off[0]; cell.g_rs = s.n[3]; cell.r_off = s.off[1]; cell.i_off = s.off[2]; cell.g_bw = s.n[4]; cell.g_bs = s.n[5];
                cell.y_rs = s.n[6]; cell.y_off = s.off[3]; cell.rb_off = s.off[4]; cell.ib_off = s.off[5]; cell.lam_off = s.off[6]; cell.act = s.n[9]; cell.c = s.f[0];
                launch_pdl_if(T < (uint32_t)kLongWalk, k_channel_scan<RgLruCell<WT>>, dim3((s.n[1] + kGruChannels - 1) / kGruChannels), dim3(kGruChannels, n_seg), 0, st, cell, bufs[s.buf[0]],
                              bufs[s.buf[5]], (const float*)bufs[s.buf[6]], T, s.n[1], s.n[7], seg_len);
            });
            ZG_SEQ_CHECK();
            return true;
        }
        case ZG_OP_GATED_NORM: {
            const uint32_t gs = s.n[1] / s.n[2];
            const uint32_t threads = gs <= 64 ? 32 : (gs <= 1024 ? 128 : (gs <= 2048 ? 256 : 512));   // at most 8 values per thread up to 4096 columns
            ZG_SEQ_WDT(s.n[4], launch_pdl(k_gated_norm<WT>, dim3(s.n[0] * s.n[2]), dim3(threads), 0, st, bufs[s.buf[0]], bufs[s.buf[1]], bufs[s.buf[2]] + s.off[0],
                                          wptr<WT>(bufs, s.buf[3], s.off[1]), s.n[1], s.n[2], s.n[3], s.n[5], s.n[6], s.f[0], s.n[7]));
            ZG_SEQ_CHECK();
            return true;
        }
        case ZG_OP_HEAD_NORM: {
            const uint32_t items = s.n[0] * s.n[1];
            ZG_SEQ_WDT(s.n[4], launch_pdl(k_head_norm<WT>, dim3((items + 3) / 4), dim3(128), 0, st, bufs[s.buf[0]] + s.off[0], wptr<WT>(bufs, s.buf[1], s.off[1]), bufs[s.buf[2]], s.n[0], s.n[1],
                                          s.n[2], s.n[3], s.n[5], s.f[0], s.f[1]));
            ZG_SEQ_CHECK();
            return true;
        }
        case ZG_OP_ACTIVATION:
            if (s.n[0] % 4 == 0 && ((reinterpret_cast<uintptr_t>(bufs[s.buf[0]]) | reinterpret_cast<uintptr_t>(bufs[s.buf[1]])) & 15) == 0)
                launch_pdl(k_activation<true>, dim3((s.n[0] / 4 + 255) / 256), dim3(256), 0, st, bufs[s.buf[0]], (const float*)bufs[s.buf[1]], s.n[0], s.n[1], s.f[0]);
            else
                launch_pdl(k_activation<false>, dim3((s.n[0] + 255) / 256), dim3(256), 0, st, bufs[s.buf[0]], (const float*)bufs[s.buf[1]], s.n[0], s.n[1], s.f[0]);
            ZG_SEQ_CHECK();
            return true;
        default:
            zg_set_error("unsupported sequence op tag %u", op.tag);
            return false;
    }
}
