// Quantized matmul of three to eight activation rows in one pass over the weight records (zg_internal.cuh), HBM-bound by intent.
//
// The arithmetic is the decode matvec's (qgemv.cu): c[m, k] = x[m, k] * s[k, nb] on a 23-bit grid per (row, quant block, warp's k-range), three base-256 digits
// of it times the raw integer weights on the integer tensor cores, exact sums, a column of ones to take the digits' offset away.  What differs is where a
// digit comes from.  The B operand of mma.sync.m16n8k32 wants, in lane 4 g + t, column g's bytes for k = 4 t .. + 3 and 16 + 4 t .. + 3.  With a column per
// ACTIVATION ROW and an MMA per digit, the lane that owns (row g, those eight k) forms their digits itself: eight scales (one 16-byte read: the records keep
// them in this order), eight staged activations (two reads), eight FMAs, twelve byte permutations, and the three operands are in its registers.  Digit
// planes in shared memory, a column per (row, digit), cost 129 warp instructions a record for four rows and two passes over the weights for more than four:
// 6 rows against two Q8_0 matrices of 14336 x 4096 took 72 us; this form takes 33 (about 45 instructions a record for any number of rows up to eight).
//
// Work split: CTA = (P column groups) x (one of S k-splits); its 16 warps split the k-range, at most eight records each, so that a row's grid is made for at most
// 256 activations; up to 64 records of K two teams of eight warps take every other column group each.  Per column group the warps' sums are added in shared memory
// in fixed order.  With S > 1 the CTAs of a column group are a cluster (S = 2, 4, 8) and add their sums over distributed shared memory, several column groups at a
// time, or meet in global scratch.
// The C operand leaves all three digits of (column g, rows 2 t and 2 t + 1) in one lane: they are put together without shuffles.
#include "split_tc.cuh"

#include <algorithm>
#include <string.h>

namespace {

constexpr uint32_t kRowsWarps = 16, kRowsThreads = 32 * kRowsWarps, kRowsCap = 8;      // records a warp stages activations for
constexpr uint32_t kRowsSmem = 205056;                                                 // eight rows of eight records of the widest format: 227 KB with the static part
constexpr uint32_t kRowsHeld = 8;                                                      // column groups whose sums wait for the cluster
constexpr uint32_t kRowsPitch = 36;                                                    // floats of a row of 32 partial sums: rows 2 t of a store in different banks

struct RowsParams {
    const uint8_t* recs;
    const float* smax;
    const float* x;
    float* out;
    float* partials;
    uint32_t* counters;
    uint32_t n_kc, n_nb, K, M, x_rs, out_rs, P, S, NS, cl, L;      // L: records of activations staged per warp
};
struct RowsBatch { RowsParams p[kZgGemvBatch]; };

__device__ __forceinline__ void imma_s8u8(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void imma_u8u8(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 rows_lds128(uint32_t addr) {
    uint4 r;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(addr));
    return r;
}
__device__ __forceinline__ void rows_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// digits 0, 1, 2 of four values: their low three bytes, a word of four per digit
__device__ __forceinline__ void digits4(const float (&F)[4], uint32_t (&d)[3]) {
    const uint32_t f0 = __float_as_uint(F[0]), f1 = __float_as_uint(F[1]), f2 = __float_as_uint(F[2]), f3 = __float_as_uint(F[3]);
    const uint32_t a01 = __byte_perm(f0, f1, 0x5140), a23 = __byte_perm(f2, f3, 0x5140);
    d[0] = __byte_perm(a01, a23, 0x5410);
    d[1] = __byte_perm(a01, a23, 0x7632);
    d[2] = __byte_perm(__byte_perm(f0, f1, 0x0062), __byte_perm(f2, f3, 0x0062), 0x5410);
}

template <int FMT, int TEAMS>
__global__ void __launch_bounds__(kRowsThreads, 1) qgemv_rows_kernel(const __grid_constant__ RowsBatch bt) {
    const RowsParams& p = bt.p[blockIdx.y];
    constexpr bool kI4 = FMT == ZG_QFMT_I4_F16, kF32 = FMT == ZG_QFMT_I8_F32;
    constexpr uint32_t QB = kI4 ? 512u : 1024u, RB = QB + (kF32 ? 128u : 64u), G = kI4 ? 4u : 2u;      // bytes of a record; records of a slot
    __shared__ float part[kRowsWarps][8][kRowsPitch];
    __shared__ float xpart[TEAMS == 1 ? kRowsHeld : 1][8][ZG_TN];
    __shared__ uint32_t s_last;
    extern __shared__ __align__(128) uint8_t dsm[];      // [warp][slot][G records] | [warp][row][L records of 32] | [warp][slot] mbarriers
    constexpr uint32_t W = kRowsWarps / TEAMS;           // warps of a team
    const uint32_t tid = threadIdx.x % (32 * W), lane = tid & 31, warp = threadIdx.x >> 5, team = TEAMS == 1 ? 0 : threadIdx.x / (32 * W), g = lane >> 2, t = lane & 3, of_team = warp % W;
    auto sync = [&] { if (TEAMS == 1) __syncthreads(); else bar_sync(1 + team, 32 * W); };
    const uint32_t split = blockIdx.x % p.S, grp = blockIdx.x / p.S, nb_begin = grp * p.P, nb_end = min(nb_begin + p.P, p.n_nb);
    const uint32_t ks = (uint32_t)(((uint64_t)split * p.n_kc) / p.S), ke = (uint32_t)(((uint64_t)(split + 1) * p.n_kc) / p.S);
    const uint32_t k0 = ks + of_team * (ke - ks) / W, L = ks + (of_team + 1) * (ke - ks) / W - k0;      // this warp's records of a column group
    const uint32_t NS = p.NS, n_chunk = (L + G - 1) / G, row_elems = p.L * ZG_KR;
    const uint32_t ring = smem_u32(dsm) + warp * NS * G * RB;
    float* xs = reinterpret_cast<float*>(dsm + kRowsWarps * NS * G * RB) + (size_t)warp * p.M * row_elems;
    const uint32_t bars = smem_u32(dsm) + kRowsWarps * (NS * G * RB + p.M * row_elems * 4) + warp * NS * 8;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    // weights are immutable: the first NS slots are asked for before the wait on the predecessor
    const uint32_t nb0 = nb_begin + team;
    uint32_t ask_c = 0, ask_slot = 0, ask_left = nb0 < nb_end ? n_chunk * ((nb_end - nb0 + TEAMS - 1) / TEAMS) : 0;
    const uint8_t* ask_src = p.recs + ((size_t)nb0 * p.n_kc + k0) * RB;
    auto ask = [&] {                                     // lane 0
        const uint32_t bytes = min(G, L - ask_c * G) * RB, bar = bars + ask_slot * 8;
        mbar_expect_tx(bar, bytes);
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"(ring + ask_slot * G * RB), "l"(ask_src + (size_t)ask_c * G * RB), "r"(bytes), "r"(bar) : "memory");
        ask_left--;
        if (++ask_c == n_chunk) { ask_c = 0; ask_src += (size_t)p.n_kc * RB * TEAMS; }
        if (++ask_slot == NS) ask_slot = 0;
    };
    if (lane == 0) {
        for (uint32_t s = 0; s < NS; s++) mbar_init(bars + s * 8, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (uint32_t i = 0; i < NS && ask_left; i++) ask();
    }
    __syncwarp();
    float sm = __ldg(p.smax + min(nb0, p.n_nb - 1)), sm_next = sm;   // power of two >= every scale of the column group
    asm volatile("griddepcontrol.wait;" ::: "memory");
    // x'[m, k] = x[m, k] * 0.499 / (max|x| * smax) of this warp's k-range (so that |s x'| <= 0.499); the four-value groups of odd rows change halves (banks of the
    // reads below).  Rows that are not finite poison their sums.
    float amax0 = 0.0f, amax1 = 0.0f;                    // max|x| of the rows 2 t and 2 t + 1, whose sums this lane holds
    {
        const uint32_t kb = k0 * ZG_KR;
        const float rsm = 1.0f / sm;
        for (uint32_t m0 = 0; m0 < p.M; m0 += 4) {       // four rows' loads in flight at once
            float v[4][kRowsCap];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float* xr = p.x + (size_t)min(m0 + j, p.M - 1) * p.x_rs + kb + lane;
#pragma unroll
                for (int i = 0; i < (int)kRowsCap; i++) v[j][i] = (uint32_t)i < L && kb + lane + 32 * i < p.K ? xr[32 * i] : 0.0f;
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const uint32_t m = m0 + j;
                if (m >= p.M) break;
                float mx = 0.0f;
#pragma unroll
                for (int i = 0; i < (int)kRowsCap; i++) { const float a = fabsf(v[j][i]); mx = a <= 3.0e38f ? fmaxf(mx, a) : INFINITY; }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                if (m == 2 * t) amax0 = mx;
                if (m == 2 * t + 1) amax1 = mx;
                const float f = (mx <= 3.0e38f && mx >= 1.0e-30f) ? (0.499f / mx) * rsm : 0.0f;      // tiny rows flush to zero
                float* xd = xs + m * row_elems + (lane ^ ((m & 1) << 4));
#pragma unroll
                for (int i = 0; i < (int)kRowsCap; i++)
                    if ((uint32_t)i < L) xd[32 * i] = v[j][i] * f;
            }
        }
        __syncwarp();
    }
    const uint32_t row = min(g, p.M - 1);                // columns past the last row repeat it
    const uint32_t x_lo = smem_u32(xs + row * row_elems) + 16 * (t ^ ((row & 1) << 2)), x_hi = smem_u32(xs + row * row_elems) + 16 * ((4 + t) ^ ((row & 1) << 2));
    bool ok = true;                                      // a wait that gave up: the warp's sums are not numbers (one lane's operands enter them all)
    uint32_t slot = 0, parity = 0, held = 0, half = 0;   // cluster: column groups whose sums wait, in the half of xpart at `half`
    const uint32_t hold = nb_end - nb_begin <= kRowsHeld ? kRowsHeld : kRowsHeld / 2;
    for (uint32_t nb = nb0; nb < nb_end; nb += TEAMS) {
        if (sm_next != sm) {                             // re-normalise the staged activations for this column group's scale: exact (powers of two)
            const float ratio = sm / sm_next;
            for (uint32_t i = lane; i < p.M * row_elems; i += 32) xs[i] *= ratio;
            __syncwarp();
            sm = sm_next;
        }
        if (nb + TEAMS < nb_end) sm_next = __ldg(p.smax + nb + TEAMS);
        int acc[3][2][4] = {}, ones[2][4] = {};          // [digit][column tile], and of a column of ones
        uint32_t dsum[3] = {};
        for (uint32_t c = 0; c < n_chunk; c++) {
            const uint32_t cnt = min(G, L - c * G), base = ring + slot * G * RB;
            if (!__all_sync(0xffffffffu, mbar_wait(bars + slot * 8, parity))) ok = false;
#pragma unroll
            for (uint32_t r = 0; r < G; r++) {
                if (r >= cnt) break;
                float sc[8];                             // of k = 4 t .. + 3, 16 + 4 t .. + 3
                if constexpr (kF32) {
                    const uint4 lo = rows_lds128(base + r * RB + QB + t * 32), hi = rows_lds128(base + r * RB + QB + t * 32 + 16);
                    const uint32_t w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
                    for (int i = 0; i < 8; i++) sc[i] = __uint_as_float(w[i]);
                } else {
                    const uint4 h = rows_lds128(base + r * RB + QB + t * 16);
                    const uint32_t w[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
                        sc[2 * i] = f.x; sc[2 * i + 1] = f.y;
                    }
                }
                const uint4 a0 = rows_lds128(x_lo + (c * G + r) * ZG_KR * 4), a1 = rows_lds128(x_hi + (c * G + r) * ZG_KR * 4);
                const float lo[4] = {fmaf(sc[0], __uint_as_float(a0.x), 1.5f), fmaf(sc[1], __uint_as_float(a0.y), 1.5f), fmaf(sc[2], __uint_as_float(a0.z), 1.5f), fmaf(sc[3], __uint_as_float(a0.w), 1.5f)};
                const float hi[4] = {fmaf(sc[4], __uint_as_float(a1.x), 1.5f), fmaf(sc[5], __uint_as_float(a1.y), 1.5f), fmaf(sc[6], __uint_as_float(a1.z), 1.5f), fmaf(sc[7], __uint_as_float(a1.w), 1.5f)};
                uint32_t b0[3], b1[3];
                digits4(lo, b0);
                digits4(hi, b1);
                uint32_t a[2][4];
                const uint4 q0 = rows_lds128(base + r * RB + lane * 16);
                if constexpr (kI4) {                     // row g: 16 u[n + 8] + u[n], row g + 8: u[n]
                    a[0][0] = q0.x; a[0][1] = q0.x & 0x0F0F0F0Fu; a[0][2] = q0.y; a[0][3] = q0.y & 0x0F0F0F0Fu;
                    a[1][0] = q0.z; a[1][1] = q0.z & 0x0F0F0F0Fu; a[1][2] = q0.w; a[1][3] = q0.w & 0x0F0F0F0Fu;
                } else {
                    const uint4 q1 = rows_lds128(base + r * RB + 512 + lane * 16);
                    a[0][0] = q0.x; a[0][1] = q0.y; a[0][2] = q0.z; a[0][3] = q0.w;
                    a[1][0] = q1.x; a[1][1] = q1.y; a[1][2] = q1.z; a[1][3] = q1.w;
                }
#pragma unroll
                for (int ct = 0; ct < 2; ct++) {
#pragma unroll
                    for (int j = 0; j < 3; j++) {
                        if constexpr (kI4) imma_u8u8(acc[j][ct], a[ct], b0[j], b1[j]);
                        else imma_s8u8(acc[j][ct], a[ct], b0[j], b1[j]);
                    }
                    if constexpr (kI4) imma_u8u8(ones[ct], a[ct], 0x01010101u, 0x01010101u);
                    else imma_s8u8(ones[ct], a[ct], 0x01010101u, 0x01010101u);
                }
                if constexpr (kI4) {
#pragma unroll
                    for (int j = 0; j < 3; j++) dsum[j] = __dp4a(b0[j], 0x01010101u, __dp4a(b1[j], 0x01010101u, dsum[j]));
                }
            }
            __syncwarp();                                // everyone is done with the slot
            if (lane == 0 && ask_left) ask();
            if (++slot == NS) { slot = 0; parity ^= 1; }
        }
        // integer sums -> this warp's partial sums.  2^-23 E2, E2 = max|x| smax / 0.499
        float esc[2];
        long long dS[2] = {0, 0};
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const float xw = i ? amax1 : amax0;
            esc[i] = xw <= 3.0e38f && ok ? (xw >= 1.0e-30f ? (xw * (2.004008016f * 1.1920928955078125e-07f)) * sm : 0.0f) : __int_as_float(0x7fc00000);
        }
        if constexpr (kI4) {
#pragma unroll
            for (int j = 0; j < 3; j++) {
                uint32_t d = dsum[j];                    // of row g
                d += __shfl_xor_sync(0xffffffffu, d, 1);
                d += __shfl_xor_sync(0xffffffffu, d, 2);
#pragma unroll
                for (int i = 0; i < 2; i++) dS[i] += (long long)__shfl_sync(0xffffffffu, d, 4 * (2 * t + i)) << (8 * j);
            }
        }
#pragma unroll
        for (int ct = 0; ct < 2; ct++)
#pragma unroll
            for (int i = 0; i < 2; i++)                  // rows 2 t and 2 t + 1
#pragma unroll
                for (int h = 0; h < 2; h++) {            // columns g and g + 8
                    long long T;
                    if constexpr (!kI4) {
                        T = (long long)acc[0][ct][2 * h + i] + ((long long)acc[1][ct][2 * h + i] << 8) + ((long long)acc[2][ct][2 * h + i] << 16) - 12582912LL * (long long)ones[ct][2 * h + i];
                    } else {                             // Y (row g + 8) = sum u[n] d, X (row g) = sum (16 u[n + 8] + u[n]) d
                        auto u = [&](const int (&o)[4]) { return (long long)(h ? (o[i] - o[2 + i]) >> 4 : o[2 + i]); };
                        T = u(acc[0][ct]) + (u(acc[1][ct]) << 8) + (u(acc[2][ct]) << 16) - 8 * dS[i] - 12582912LL * (u(ones[ct]) - 8LL * (long long)(L * ZG_KR));
                    }
                    part[warp][2 * t + i][ct * 16 + g + 8 * h] = __ll2float_rn(T) * esc[i];
                }
        sync();
        const uint32_t m = tid >> 5, col = tid & 31;
        float v = 0.0f;
        if (m < p.M) {
#pragma unroll
            for (uint32_t w = 0; w < W; w++) v += part[team * W + w][m][col];
            if (p.S == 1) p.out[(size_t)m * p.out_rs + nb * ZG_TN + col] = v;
            else if (p.cl) xpart[half + held][m][col] = v;
            else p.partials[(((size_t)nb * p.S + split) * 8 + m) * ZG_TN + col] = v;
        }
        sync();                                          // the sums are read: the next column group may overwrite them
        if (TEAMS == 1 && p.S > 1 && p.cl) {
            if (++held < hold && nb + 1 < nb_end) continue;
            // One cluster barrier publishes the partial sums of these column groups; the CTAs of the cluster take them in turns and add them in split order.  The next ones
            // use the other half, and whoever reads reaches the barrier after that only when it has read.
            rows_cluster_sync();
            for (uint32_t i = split; i < held; i += p.S) {
                if (m >= p.M) break;
                v = 0.0f;
                for (uint32_t s2 = 0; s2 < p.S; s2++) {
                    uint32_t remote; float x;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(&xpart[half + i][m][col])), "r"(s2));
                    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x) : "r"(remote) : "memory");
                    v += x;
                }
                p.out[(size_t)m * p.out_rs + (nb + 1 - held + i) * ZG_TN + col] = v;
            }
            held = 0;
            half ^= kRowsHeld / 2;
        } else if (TEAMS == 1 && p.S > 1) {
            if (tid == 0) {
                uint32_t old;
                asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(p.counters + nb) : "memory");
                s_last = old == p.S - 1 ? 1u : 0u;
                if (old == p.S - 1) p.counters[nb] = 0u; // re-arm for the next launch
            }
            __syncthreads();
            if (s_last && m < p.M) {
                v = 0.0f;
                for (uint32_t s2 = 0; s2 < p.S; s2++) v += __ldcg(p.partials + (((size_t)nb * p.S + s2) * 8 + m) * ZG_TN + col);
                p.out[(size_t)m * p.out_rs + nb * ZG_TN + col] = v;
            }
        }
    }
    if (!ok && lane == 0) count_timeout();
    if (TEAMS == 1 && p.S > 1 && p.cl) rows_cluster_sync();      // nobody leaves while another may still read its partials
}

template <int FMT, int TEAMS>
bool launch_teams(const ZgGemvRowsPlan& pl, const RowsBatch& bt, uint32_t count, bool cluster, bool pdl, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(pl.grid, count);
    cfg.blockDim = dim3(kRowsThreads);
    cfg.dynamicSmemBytes = pl.smem_bytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    unsigned na = 0;
    if (pdl) { attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization; attr[na].val.programmaticStreamSerializationAllowed = 1; na++; }
    if (cluster) { attr[na].id = cudaLaunchAttributeClusterDimension; attr[na].val.clusterDim.x = pl.S; attr[na].val.clusterDim.y = 1; attr[na].val.clusterDim.z = 1; na++; }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    if (!zg_smem_limit<qgemv_rows_kernel<FMT, TEAMS>>(kRowsSmem)) return false;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, qgemv_rows_kernel<FMT, TEAMS>, bt);
    ZG_COUNT_LAUNCH();
    if (e != cudaSuccess) { zg_set_error("matvec of %u rows: launch failed: %s (grid %u, %u B shared)", bt.p[0].M, cudaGetErrorString(e), pl.grid, pl.smem_bytes); return false; }
    return true;
}
template <int FMT>
bool launch_rows(const ZgGemvRowsPlan& pl, const RowsBatch& bt, uint32_t count, bool cluster, bool pdl, cudaStream_t st) {
    return pl.teams == 2 ? launch_teams<FMT, 2>(pl, bt, count, cluster, pdl, st) : launch_teams<FMT, 1>(pl, bt, count, cluster, pdl, st);
}

}  // namespace

// K is split over CTAs until a warp has at most kRowsCap records, further where the column groups would leave more than half of the SMs idle (four records a
// warp at least); then every CTA takes column groups enough that the matvecs of the launch are one wave.
ZgGemvRowsPlan zg_qgemv_rows_plan(const ZgCudaCtx* ctx, const ZgCudaQWeight* w, uint32_t M, uint32_t count) {
    ZgGemvRowsPlan pl;
    const uint32_t sms = (uint32_t)ctx->sm_count;
    pl.S = (w->n_kc + kRowsWarps * kRowsCap - 1) / (kRowsWarps * kRowsCap);
    if (w->n_nb * pl.S * 2 <= sms) pl.S = std::max(pl.S, std::min(sms / w->n_nb, w->n_kc / (kRowsWarps * 4)));
    pl.S = std::max(1u, std::min(pl.S, w->n_kc));
    pl.P = std::max(1u, (uint32_t)(((uint64_t)w->n_nb * pl.S * count + sms - 1) / sms));
    pl.grid = (w->n_nb + pl.P - 1) / pl.P * pl.S;
    pl.teams = pl.S == 1 && w->n_kc <= kRowsWarps / 2 * kRowsCap && pl.P > 1 ? 2 : 1;
    pl.L = ((w->n_kc + pl.S - 1) / pl.S + kRowsWarps / pl.teams - 1) / (kRowsWarps / pl.teams);
    const uint32_t G = w->fmt == ZG_QFMT_I4_F16 ? 4 : 2, chunks = (pl.L + G - 1) / G * ((pl.P + pl.teams - 1) / pl.teams);
    pl.NS = std::max(1u, std::min(2u, chunks));
    pl.smem_bytes = kRowsWarps * (pl.NS * G * w->rec_bytes + M * pl.L * ZG_KR * 4 + pl.NS * 8);
    return pl;
}

bool zg_qgemv_rows_launch(ZgCudaCtx* ctx, uint32_t count, const ZgCudaQWeight* const* w, const float* const* d_in, float* const* d_out, uint32_t M, const uint32_t* in_rs,
                          const uint32_t* out_rs, const ZgGemvWs* ws, cudaStream_t st) {
    const ZgCudaQWeight* w0 = w[0];
    for (uint32_t i = 1; i < count; i++) if (w[i]->N > w0->N) w0 = w[i];
    const ZgGemvRowsPlan pl = zg_qgemv_rows_plan(ctx, w0, M, count);
    const bool cluster = ctx->gemv_cluster && (pl.S == 2 || pl.S == 4 || pl.S == 8);
    RowsBatch bt;
    memset(&bt, 0, sizeof(bt));
    for (uint32_t i = 0; i < count; i++) {
        if (w[i]->fmt != w0->fmt || w[i]->K != w0->K || (w[i]->N != w0->N && pl.S > 1) || w[i]->fmt == ZG_QFMT_GENERIC) { zg_set_error("internal: mixed matvec batch"); return false; }
        size_t pe = 0, nc = 0;
        zg_qgemv_ws_need(ctx, w[i], M, &pe, &nc);
        if (pe && (ws[i].partials_elems < pe || ws[i].counters_n < nc)) { zg_set_error("internal: split workspace too small (%zu/%zu needed)", pe, nc); return false; }
        bt.p[i] = {w[i]->recs, w[i]->smax, d_in[i], d_out[i], ws[i].partials, ws[i].counters, w[i]->n_kc, w[i]->n_nb, (uint32_t)w[i]->K, M, in_rs[i] ? in_rs[i] : (uint32_t)w[i]->K,
                   out_rs[i] ? out_rs[i] : (uint32_t)w[i]->N, pl.P, pl.S, pl.NS, cluster ? 1u : 0u, pl.L};
    }
    switch (w[0]->fmt) {
        case ZG_QFMT_I8_F32: return launch_rows<ZG_QFMT_I8_F32>(pl, bt, count, cluster, ctx->pdl, st);
        case ZG_QFMT_I8_F16: return launch_rows<ZG_QFMT_I8_F16>(pl, bt, count, cluster, ctx->pdl, st);
        case ZG_QFMT_I4_F16: return launch_rows<ZG_QFMT_I4_F16>(pl, bt, count, cluster, ctx->pdl, st);
        default: zg_set_error("qmatmul: unknown weight format %d", w[0]->fmt); return false;
    }
}
unsigned int zg_qgemv_rows_timeouts() { return tc_timeouts(); }
