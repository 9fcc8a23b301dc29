// LINEAR of many rows over f32 weights on the tensor cores, with f32 accuracy:  part[m, n] = sum_k src[m, k] W[n, k].
//
// Both operands are cut into three bfloat16 parts inside the kernel, 64 k at a time: b0 = bf16(x), b1 = bf16(x - b0), b2 = x - b0 - b1.  Three 8-bit
// significands hold all 24 bits of x, and every part has an f32's range of exponents: nothing is scaled, and what one element of a row keeps does not
// depend on the others (pairs of half precision with a scale per row and 64 k, three MMAs a product, lost the small elements beside a large one and
// left f32's range before the scales were undone).  Below 2^-109 the last part runs out of exponents: such an element is held to 2^-134.
// A product is the six MMAs b1 b1 + b0 b2 + b2 b0 + b0 b1 + b1 b0 + b0 b0, the smallest first; what is left out (b1 b2 and smaller) is at most 2^-23 of it,
// 2^-26 on average.
// The tensor core's f32 accumulator truncates, which over a long sum would cost more than an f32 chain rounds, so it holds the products of ONE 64-k step
// (four additions of b0 b0) and the steps are added in registers in f32.  Error against 64 bits at 256 tokens, 2048 / 4096: 1.7e-7 (pairs 2.1e-7, the f32
// tile 8.7e-7).
//
//   * 128 x 128 tile per CTA, grid (n tiles, m tiles, shares of K).  Sixteen worker warps load f32 rows of the weights (16 lanes per row of 64), two steps ahead, cut
//     them, and store swizzled K-major tiles into a 2-stage ring; the same warps drain the accumulators of the step before (two TMEM buffers), each a quarter of
//     the columns of its 32 rows.  Warp 16 issues the MMAs, warp 17 brings the source's parts, which k_split_source has cut once for all tiles of weight rows.
//   * Per step the MMAs take 1536 clocks, their operand reads, the copies and the stores 2300 clocks of shared-memory bandwidth.  Where the workers cut the source
//     too, every CTA its 128 rows of it, a step was 555 instructions of each worker warp, 2200 clocks of issue and 5000 in all, with its loads in flight for one step
//     only: 256 tokens through gate, up and down of 2048 / 4096 took 166 us, now 105 (as the f32 tile 1034).
//   * One share of K: the tile is finished here (bias, activation) and leaves by whole rows.  Several: partial sums go to scratch and k_split_finish adds them in
//     order.  A sum that is not finite is evaluated again as a plain f32 sum: what an infinity makes of a sum is the plain kernel's.
//   * Every wait is bounded and counts itself (with the count after the loops the case above took 178 us); a CTA whose wait ran out treats its sums as
//     not finite, so that they are evaluated again the plain way.
#include "split_tc.cuh"

#include <algorithm>
#include <string.h>

namespace {

constexpr uint32_t kBM = 128, kBN = 128, kBK = 64;
constexpr uint32_t kTile = kBM * kBK * 2, kSgStage = 6 * kTile, kSgStages = 2, kSgWorkers = 512;
constexpr uint32_t kSgSmem = kSgStages * kSgStage + 1024 + 128;

struct SgArgs {
    const float* src; const float* W; float* part;
    uint32_t M, N, K, src_rs, part_rs, splits;       // N: weight rows
    const float* ctl; uint32_t slot_stride, rows_from;
    float* dst; const float* bias; uint32_t dst_rs, pairs; SeqAct act;
    uint16_t* planes; uint32_t pitch;                // PRE: [part][M][pitch] bfloat16 of the source
};
__device__ __forceinline__ const float* sg_src(const SgArgs& a) { return a.src + (a.ctl && a.slot_stride ? (size_t)ctl_word(a.ctl, ZG_CTL_SLOT) * a.slot_stride : 0); }
__device__ __forceinline__ float plain_sum(const float* x, const float* w, uint32_t K) {
    float acc = 0.0f;
#pragma unroll 1
    for (uint32_t k = 0; k < K; k++) acc = fmaf(x[k], w[k], acc);
    return acc;
}
// sums of four weight rows n .. n + 3 of source row m -> bias, activation, dst (pairs: two outputs)
__device__ __forceinline__ void sg_finish(const SgArgs& a, uint32_t m, uint32_t n, float4 v) {
    float z[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; j++)
        if (!(fabsf(z[j]) <= 3.4028234e38f) && n + j < a.N) z[j] = plain_sum(sg_src(a) + (size_t)m * a.src_rs, a.W + (size_t)(n + j) * a.K, a.K);
    float* out = a.dst + (size_t)m * a.dst_rs;
    if (a.pairs) {
#pragma unroll
        for (int j = 0; j < 4; j += 2) if (n + j + 1 < a.N) out[(n + j) / 2] = seq_epilogue(z[j], a.act.kind, a.act.p) * z[j + 1];
        return;
    }
#pragma unroll
    for (int j = 0; j < 4; j++)
        if (n + j < a.N) z[j] = seq_epilogue(z[j] + (a.bias ? a.bias[n + j] : 0.0f), a.act, n + j);
    if (n + 4 <= a.N && (reinterpret_cast<uintptr_t>(out + n) & 15) == 0) *reinterpret_cast<float4*>(out + n) = make_float4(z[0], z[1], z[2], z[3]);
    else
        for (int j = 0; j < 4; j++) if (n + j < a.N) out[n + j] = z[j];
}

// The source's parts, once per linear instead of once per tile of weight rows: eight elements a thread.  Where only the rows that a sequence holds count, the row tiles
// that hold some (8192 rows of 576 at position 100, 1024 outputs: 23.3 us with all rows cut, 18.3; of 512 and 4096 outputs 37.5, 32.2).
__global__ void __launch_bounds__(256) k_split_source(const SgArgs a) {
    pdl_enter();
    const float* src = sg_src(a);
    const uint32_t per_row = a.pitch / 8, rows = a.rows_from ? min(a.M, ((uint32_t)ctl_word(a.ctl, ZG_CTL_POS) + a.rows_from + kBM - 1) / kBM * kBM) : a.M;
    for (size_t e = blockIdx.x * 256 + threadIdx.x; e < (size_t)rows * per_row; e += (size_t)gridDim.x * 256) {
        const uint32_t m = (uint32_t)(e / per_row), k = (uint32_t)(e % per_row) * 8;
        const float* x = src + (size_t)m * a.src_rs + k;      // K is a multiple of four
        const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f), u = *reinterpret_cast<const float4*>(x), v = k + 4 < a.K ? *reinterpret_cast<const float4*>(x + 4) : zero;
        uint4 p[3];
        split3(u.x, u.y, p[0].x, p[1].x, p[2].x);
        split3(u.z, u.w, p[0].y, p[1].y, p[2].y);
        split3(v.x, v.y, p[0].z, p[1].z, p[2].z);
        split3(v.z, v.w, p[0].w, p[1].w, p[2].w);
#pragma unroll
        for (int i = 0; i < 3; i++) *reinterpret_cast<uint4*>(a.planes + ((size_t)i * a.M + m) * a.pitch + k) = p[i];
    }
}

// PRE: the source's parts come by TMA from k_split_source's planes (warp 17), the workers cut the weights alone and load them two steps ahead
template <bool PRE>
__global__ void __launch_bounds__(kSgWorkers + (PRE ? 64 : 32), 1) k_split_gemm(const SgArgs a, const __grid_constant__ CUtensorMap planes) {
    extern __shared__ uint8_t dsm_raw[];
    const uint32_t base = (smem_u32(dsm_raw) + 1023u) & ~1023u, bars = base + kSgStages * kSgStage;
    const uint32_t full = bars, empty = full + 8 * kSgStages, d_full = empty + 8 * kSgStages, d_empty = d_full + 16, tmem_slot = d_empty + 16;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < kSgStages; i++) { mbar_init(full + 8 * i, PRE ? 17 : 16); mbar_init(empty + 8 * i, 1); }
        for (uint32_t i = 0; i < 2; i++) { mbar_init(d_full + 8 * i, 1); mbar_init(d_empty + 8 * i, 16); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 16) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" ::"r"(tmem_slot) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    uint32_t tmem;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(tmem_slot));
    tmem = __shfl_sync(0xffffffffu, tmem, 0);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t m0 = blockIdx.y * kBM, n0 = blockIdx.x * kBN, steps = (a.K + kBK - 1) / kBK;
    const uint32_t s0 = (uint32_t)((uint64_t)blockIdx.z * steps / a.splits), s1 = (uint32_t)((uint64_t)(blockIdx.z + 1) * steps / a.splits);
    const bool live = !(a.rows_from && m0 >= (uint32_t)ctl_word(a.ctl, ZG_CTL_POS) + a.rows_from);
    const uint32_t n_steps = live ? s1 - s0 : 0;

    if (warp == 16) {
        constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((kBN >> 3) << 17) | ((kBM >> 4) << 24);       // bf16 x bf16 -> f32
        const bool leader = elect_one();
        const uint32_t b0 = desc_low(base);
        bool ok = true;
        uint32_t stage = 0, phase = 0;
        for (uint32_t i = 0; i < n_steps; i++) {
            if (ok) ok = mbar_wait_counted(full + 8 * stage, phase);
            if (ok && i >= 2) ok = mbar_wait_counted(d_empty + 8 * (i & 1), ((i >> 1) - 1) & 1);
            fence_after();
            if (leader && ok) {
                const uint32_t d = tmem + (i & 1) * kBN, x0 = b0 + stage * (kSgStage >> 4);
                constexpr uint32_t kPart[6][2] = {{1, 1}, {0, 2}, {2, 0}, {0, 1}, {1, 0}, {0, 0}};       // parts of the source, of the weights
#pragma unroll
                for (uint32_t p = 0; p < 6; p++)
#pragma unroll
                    for (uint32_t k = 0; k < 4; k++) {
                        const uint32_t x = x0 + kPart[p][0] * (kTile >> 4) + 2 * k, w = x0 + (3 + kPart[p][1]) * (kTile >> 4) + 2 * k;
                        if (p == 0 && k == 0) mma_ss<false>(d, x, w, idesc); else mma_ss<true>(d, x, w, idesc);
                    }
                mma_commit(empty + 8 * stage);
                mma_commit(d_full + 8 * (i & 1));
            }
            __syncwarp();
            if (++stage == kSgStages) { stage = 0; phase ^= 1; }
        }
    } else if (PRE && warp == 17) {
        bool ok = true;
        uint32_t stage = 0, phase = 1;
        for (uint32_t i = 0; i < n_steps && ok; i++) {
            ok = mbar_wait_counted(empty + 8 * stage, phase);
            if (lane == 0 && ok) {
                mbar_expect_tx(full + 8 * stage, 3 * kTile);
                const int32_t k = (int32_t)((s0 + i) * kBK), m = (int32_t)m0;
                asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                             ::"r"(base + stage * kSgStage), "l"(&planes), "r"(k), "r"(m), "r"(0), "r"(full + 8 * stage) : "memory");
            }
            __syncwarp();
            if (++stage == kSgStages) { stage = 0; phase ^= 1; }
        }
    } else {
        // loading: lane group of 16 takes rows r + 32 i, columns 4 c .. + 3 of a step; draining: rows of the warp's quarter, 32 columns
        const uint32_t c = threadIdx.x & 15, r = threadIdx.x >> 4, quarter = warp & 3, part = warp >> 2;
        uint8_t* const ring = dsm_raw + (base - smem_u32(dsm_raw));
        const float* src = sg_src(a);
        constexpr int FIRST = PRE ? 4 : 0, AHEAD = PRE ? 2 : 1;
        float4 x[AHEAD][8];                                          // four rows of the source, four of the weights
        auto load = [&](uint32_t step, float4 (&x)[8]) {
            const uint32_t k = step * kBK + 4 * c;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t m = m0 + r + 32 * i, n = n0 + r + 32 * i;
                if (!PRE) x[i] = m < a.M && k < a.K ? *reinterpret_cast<const float4*>(src + (size_t)m * a.src_rs + k) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                x[4 + i] = n < a.N && k < a.K ? *reinterpret_cast<const float4*>(a.W + (size_t)n * a.K + k) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
        };
        float acc[32];
#pragma unroll
        for (int j = 0; j < 32; j++) acc[j] = 0.0f;
        bool ok = true;
        auto drain = [&](uint32_t i) {
            if (ok) ok = __all_sync(0xffffffffu, mbar_wait_counted(d_full + 8 * (i & 1), (i >> 1) & 1));
            fence_after();
#pragma unroll
            for (int h = 0; h < 32; h += 16) {                       // half at a time: the registers of the other half hold rows on their way
                uint32_t v[16];
                tmem_ld(tmem + ((quarter * 32) << 16) + (i & 1) * kBN + 32 * part + h, v);
                tmem_wait_ld(v);
                if (h) {
                    fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(d_empty + 8 * (i & 1));
                }
#pragma unroll
                for (int j = 0; j < 16; j += 2) {
                    const float2 r = __fadd2_rn(make_float2(acc[h + j], acc[h + j + 1]), make_float2(__uint_as_float(v[j]), __uint_as_float(v[j + 1])));
                    acc[h + j] = r.x; acc[h + j + 1] = r.y;
                }
            }
        };
        if (n_steps) load(s0, x[0]);
        if (PRE && n_steps > 1) load(s0 + 1, x[AHEAD - 1]);
        uint32_t stage = 0, phase = 1;
        auto step = [&](uint32_t i, float4 (&x)[8]) {
            if (ok) ok = __all_sync(0xffffffffu, mbar_wait_counted(empty + 8 * stage, phase));
            uint8_t* const to = ring + stage * kSgStage;
#pragma unroll
            for (int j = FIRST; j < 8; j++) {                        // the source's rows, the weights'
                const float4 y = x[j];
                const uint32_t row = r + 32 * (j & 3);
                uint2 p0, p1, p2;
                split3(y.x, y.y, p0.x, p1.x, p2.x);
                split3(y.z, y.w, p0.y, p1.y, p2.y);
                uint8_t* const at = to + (j >> 2) * 3 * kTile + row * 128 + (((c >> 1) ^ (row & 7)) * 16 + (c & 1) * 8);
                *reinterpret_cast<uint2*>(at) = p0;
                *reinterpret_cast<uint2*>(at + kTile) = p1;
                *reinterpret_cast<uint2*>(at + 2 * kTile) = p2;
            }
            if (i + AHEAD < n_steps) load(s0 + i + AHEAD, x);        // in flight while the step before is drained, and with PRE the next one is cut
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(full + 8 * stage);
            if (++stage == kSgStages) { stage = 0; phase ^= 1; }
            if (i) drain(i - 1);
        };
        for (uint32_t i = 0; i < n_steps; i += AHEAD) {
            step(i, x[0]);
            if (PRE && i + 1 < n_steps) step(i + 1, x[AHEAD - 1]);
        }
        if (n_steps) drain(n_steps - 1);
        // out by whole rows, through the idle ring (every MMA that reads it is done)
        float4* const out = reinterpret_cast<float4*>(ring);
        const uint32_t row = quarter * 32 + lane;
        bar_sync(1, kSgWorkers);
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
            const float f = ok ? 1.0f : __uint_as_float(0x7fffffffu);
            out[row * 32 + ((8 * part + j / 4) ^ (row & 7))] = make_float4(acc[j] * f, acc[j + 1] * f, acc[j + 2] * f, acc[j + 3] * f);
        }
        bar_sync(1, kSgWorkers);
        float* const p = a.part + (size_t)blockIdx.z * a.M * a.part_rs;
        for (uint32_t i = threadIdx.x; live && i < kBM * 32; i += kSgWorkers) {
            const uint32_t rr = i >> 5, j = i & 31, m = m0 + rr, n = n0 + 4 * j;
            if (m >= a.M || n >= a.N) continue;
            const float4 v = out[rr * 32 + (j ^ (rr & 7))];
            if (a.splits == 1) sg_finish(a, m, n, v);
            else *reinterpret_cast<float4*>(p + (size_t)m * a.part_rs + n) = v;
        }
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    __syncwarp();
    fence_before();
    __syncthreads();
    if (warp == 16) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(tmem) : "memory");
}

// the shares' sums, bias, activation; four weight rows per thread
__global__ void __launch_bounds__(256) k_split_finish(const SgArgs a) {
    pdl_enter();
    const uint32_t n = 4 * (blockIdx.x * 256 + threadIdx.x);
    if (n >= a.N) return;
    for (uint32_t m = blockIdx.y; m < a.M; m += gridDim.y) {
        if (a.rows_from && m / kBM * kBM >= (uint32_t)ctl_word(a.ctl, ZG_CTL_POS) + a.rows_from) return;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        for (uint32_t s = 0; s < a.splits; s++) {
            const float4 p = *reinterpret_cast<const float4*>(a.part + ((size_t)s * a.M + m) * a.part_rs + n);
            v.x += p.x; v.y += p.y; v.z += p.z; v.w += p.w;
        }
        sg_finish(a, m, n, v);
    }
}

// shares of K: the fewest rounds of CTAs times steps per CTA, a step of overhead for each round's start and end.  Several shares only where they make
// no more than four CTAs per SM, so that their partial sums stay within some 40 MB whatever the shape.
uint32_t shares(uint32_t M, uint32_t N, uint32_t K, uint32_t n_sm) {
    const uint64_t tiles = (uint64_t)((M + kBM - 1) / kBM) * ((N + kBN - 1) / kBN);
    const uint32_t steps = (K + kBK - 1) / kBK;
    uint32_t best = 1;
    uint64_t best_cost = ~0ull;
    for (uint32_t s = 1; s <= 16 && s <= (steps + 3) / 4 && (s == 1 || (uint64_t)tiles * s <= 4ull * n_sm); s++) {
        const uint64_t cost = ((tiles * s + n_sm - 1) / n_sm) * ((steps + s - 1) / s + 4) + s / 2;
        if (cost < best_cost) { best_cost = cost; best = s; }
    }
    return best;
}
uint32_t up4(uint32_t n) { return (n + 3) / 4 * 4; }
uint32_t up8(uint32_t n) { return (n + 7) / 8 * 8; }
// Whether the source is cut ahead, by a launch of its own (some 3 us): where a CTA takes four steps or more, each about 1 us shorter for it (up and down of 1000 / 3000
// with 100 tokens 58.7 us without, 43.2 from four steps on, 47.0 from eight, 51.4 always).
constexpr size_t kSgPlanes = 40u << 20;              // elements: 240 MB of planes at most
bool split_first(uint32_t M, uint32_t N, uint32_t K) {
    const uint64_t tiles = (uint64_t)((M + kBM - 1) / kBM) * ((N + kBN - 1) / kBN), n_sm = zg_sm_count();
    const uint32_t s = shares(M, N, K, (uint32_t)n_sm), steps = ((K + kBK - 1) / kBK + s - 1) / s;
    return (tiles * s + n_sm - 1) / n_sm * steps >= 4 && (size_t)M * K <= kSgPlanes && encode_tiled();
}
size_t plane_elems(uint32_t M, uint32_t N, uint32_t K) { return split_first(M, N, K) ? ((size_t)3 * M * up8(K) / 2 + 3) / 4 * 4 : 0; }

}  // namespace

// rows start at 16-byte boundaries; N counts weight rows
bool zg_split_gemm_usable(const float* w, const float* src, uint32_t M, uint32_t N, uint32_t K, uint32_t src_rs, uint32_t slot_stride) {
    return M > 8 && N >= 32 && K >= 64 && K % 4 == 0 && src_rs % 4 == 0 && slot_stride % 4 == 0 && ((reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(src)) & 15) == 0;
}
size_t zg_split_gemm_scratch_elems(uint32_t M, uint32_t N, uint32_t K, bool least) {      // never 0, which stands for the plain kernel
    const uint32_t s = shares(M, N, K, zg_sm_count());
    return (s > 1 ? (size_t)s * M * up4(N) : 4) + (least ? 0 : plane_elems(M, N, K));
}
unsigned int zg_split_gemm_timeouts() { return tc_timeouts(); }
bool zg_split_gemm_launch(const float* w, const float* bias, const float* src, float* dst, uint32_t M, uint32_t N, uint32_t K, uint32_t src_rs, uint32_t dst_rs, float* scratch, size_t scratch_elems,
                          cudaStream_t st, uint32_t act, float act_p, uint32_t act_lo, uint32_t act_hi, const float* ctl, uint32_t slot_stride, bool pairs, uint32_t rows_from) {
    if (!zg_smem_limit<k_split_gemm<false>>(kSgSmem) || !zg_smem_limit<k_split_gemm<true>>(kSgSmem)) return false;
    SgArgs a = {src, w, scratch, M, N, K, src_rs, up4(N), shares(M, N, K, zg_sm_count()), ctl, slot_stride, rows_from, dst, bias, dst_rs, (uint32_t)pairs, SeqAct{act, act_p, act_lo, act_hi}, nullptr, 0};
    const dim3 grid((N + kBN - 1) / kBN, (M + kBM - 1) / kBM, a.splits);
    CUtensorMap map;
    memset(&map, 0, sizeof(map));
    if (split_first(M, N, K) && scratch_elems >= zg_split_gemm_scratch_elems(M, N, K, false)) {      // where the planes found no room, the workers cut the source as they go
        a.planes = reinterpret_cast<uint16_t*>(scratch);
        a.pitch = up8(K);
        a.part = scratch + plane_elems(M, N, K);
        const cuuint64_t dims[3] = {a.pitch, M, 3}, strides[2] = {(cuuint64_t)a.pitch * 2, (cuuint64_t)a.pitch * 2 * M};
        const cuuint32_t box[3] = {kBK, kBM, 3}, ones[3] = {1, 1, 1};
        const CUresult r = encode_tiled()(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, a.planes, dims, strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) { zg_set_error("split gemm: tensor map failed (%d)", (int)r); return false; }
        launch_pdl(k_split_source, dim3(std::min<uint32_t>(4 * zg_sm_count(), (uint32_t)(((size_t)M * a.pitch / 8 + 255) / 256))), dim3(256), 0, st, a);
        ZG_COUNT_LAUNCH();
        launch_pdl(k_split_gemm<true>, grid, dim3(kSgWorkers + 64), kSgSmem, st, a, map);
    } else launch_pdl(k_split_gemm<false>, grid, dim3(kSgWorkers + 32), kSgSmem, st, a, map);
    ZG_COUNT_LAUNCH();
    if (a.splits > 1) {
        launch_pdl(k_split_finish, dim3((N + 1023) / 1024, M < 65535 ? M : 65535), dim3(256), 0, st, a);
        ZG_COUNT_LAUNCH();
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { zg_set_error("split gemm launch failed: %s", cudaGetErrorString(e)); return false; }
    return true;
}
