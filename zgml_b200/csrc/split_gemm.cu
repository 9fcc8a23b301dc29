// LINEAR of many rows over f32 weights on the tensor cores, with f32 accuracy:  part[m, n] = sum_k src[m, k] W[n, k].
//
// Both operands are split into half-precision pairs (split_tc.cuh) inside the kernel, 64 k at a time, each row of the 64 with a scale of its own; a product
// is three MMAs, hi lo + lo hi + hi hi.  The tensor core's f32 accumulator truncates, which over a long sum would cost more than an f32 chain
// rounds, so it holds the products of ONE 64-k step (four additions of hi hi) and the steps are added in registers in f32, with the two rows' scales
// undone on the way.
//
//   * 128 x 128 tile per CTA, grid (n tiles, m tiles, shares of K).  Sixteen worker warps load f32 rows (16 lanes per row of 64), find the row's maximum by
//     shuffles, split, and store swizzled K-major tiles into a 3-stage ring; the same warps drain the accumulators of the step before (two TMEM
//     buffers), each a quarter of the columns of its 32 rows.  Warp 16 issues the MMAs.
//   * Per step the MMAs take 768 clocks, their operand reads and the workers' stores 1280 clocks of shared-memory bandwidth, the workers' instructions
//     about 1500 issue slots per scheduler: the workers bound it.
//   * Tiles leave as partial sums; k_split_finish adds the shares in order and applies bias and activation.  A result that is not a number is evaluated
//     again there as a plain f32 sum: a row whose maximum is not finite has no scale, and what an infinity makes of a sum is the plain kernel's.
//   * Every wait is bounded; a CTA whose wait ran out writes NaN, so that its outputs are evaluated again the plain way.
#include "split_tc.cuh"

namespace {

constexpr uint32_t kBM = 128, kBN = 128, kBK = 64;
constexpr uint32_t kTile = kBM * kBK * 2, kSgStage = 4 * kTile, kSgStages = 3, kSgWorkers = 512, kSgThreads = kSgWorkers + 32;
constexpr uint32_t kSgScales = 4 * (kBM + kBN) * 4;               // of four steps: a warp may be two ahead of another's drain
constexpr uint32_t kSgSmem = kSgStages * kSgStage + kSgScales + 1024 + 128;

struct SgArgs {
    const float* src; const float* W; float* part;
    uint32_t M, N, K, src_rs, part_rs, splits;       // N: weight rows
    const float* ctl; uint32_t slot_stride, rows_from;
};

__global__ void __launch_bounds__(kSgThreads, 1) k_split_gemm(const SgArgs a) {
    extern __shared__ uint8_t dsm_raw[];
    const uint32_t base = (smem_u32(dsm_raw) + 1023u) & ~1023u, bars = base + kSgStages * kSgStage + kSgScales;
    const uint32_t full = bars, empty = full + 8 * kSgStages, d_full = empty + 8 * kSgStages, d_empty = d_full + 16, tmem_slot = d_empty + 16;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < kSgStages; i++) { mbar_init(full + 8 * i, 16); mbar_init(empty + 8 * i, 1); }
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
        constexpr uint32_t idesc = (1u << 4) | ((kBN >> 3) << 17) | ((kBM >> 4) << 24);       // f16 x f16 -> f32
        const bool leader = elect_one();
        const uint32_t b0 = desc_low(base);
        bool ok = true;
        uint32_t stage = 0, phase = 0;
        for (uint32_t i = 0; i < n_steps; i++) {
            if (ok) ok = mbar_wait(full + 8 * stage, phase);
            if (ok && i >= 2) ok = mbar_wait(d_empty + 8 * (i & 1), ((i >> 1) - 1) & 1);
            fence_after();
            if (leader && ok) {
                const uint32_t d = tmem + (i & 1) * kBN, ah = b0 + stage * (kSgStage >> 4), al = ah + (kTile >> 4), bh = al + (kTile >> 4), bl = bh + (kTile >> 4);
                mma_ss<false>(d, ah, bl, idesc);
#pragma unroll
                for (uint32_t k = 1; k < 4; k++) mma_ss<true>(d, ah + 2 * k, bl + 2 * k, idesc);
#pragma unroll
                for (uint32_t k = 0; k < 4; k++) mma_ss<true>(d, al + 2 * k, bh + 2 * k, idesc);
#pragma unroll
                for (uint32_t k = 0; k < 4; k++) mma_ss<true>(d, ah + 2 * k, bh + 2 * k, idesc);
                mma_commit(empty + 8 * stage);
                mma_commit(d_full + 8 * (i & 1));
            }
            __syncwarp();
            if (++stage == kSgStages) { stage = 0; phase ^= 1; }
        }
    } else {
        // loading: lane group of 16 takes rows r + 32 i, columns 4 c .. + 3 of a step; draining: rows of the warp's quarter, 32 columns
        const uint32_t c = threadIdx.x & 15, r = threadIdx.x >> 4, quarter = warp & 3, part = warp >> 2;
        uint8_t* const ring = dsm_raw + (base - smem_u32(dsm_raw));
        float* const scales = reinterpret_cast<float*>(ring + kSgStages * kSgStage);
        const float* src = a.src + (a.ctl && a.slot_stride ? (size_t)ctl_word(a.ctl, ZG_CTL_SLOT) * a.slot_stride : 0);
        float4 x[8];                                                 // four rows of the source, four of the weights
        auto load = [&](uint32_t step) {
            const uint32_t k = step * kBK + 4 * c;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t m = m0 + r + 32 * i, n = n0 + r + 32 * i;
                x[i] = m < a.M && k < a.K ? *reinterpret_cast<const float4*>(src + (size_t)m * a.src_rs + k) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                x[4 + i] = n < a.N && k < a.K ? *reinterpret_cast<const float4*>(a.W + (size_t)n * a.K + k) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
        };
        float acc[32];
#pragma unroll
        for (int j = 0; j < 32; j++) acc[j] = 0.0f;
        bool ok = true;
        auto drain = [&](uint32_t i) {
            if (ok) ok = __all_sync(0xffffffffu, mbar_wait(d_full + 8 * (i & 1), (i >> 1) & 1));
            fence_after();
            uint32_t v[32];
            tmem_ld(tmem + ((quarter * 32) << 16) + (i & 1) * kBN + 32 * part, v);
            tmem_wait_ld(v);
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(d_empty + 8 * (i & 1));
            const float* sc = scales + (i & 3) * (kBM + kBN);
            const float sa = sc[quarter * 32 + lane];
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
                const float4 sb = *reinterpret_cast<const float4*>(sc + kBM + 32 * part + j);
                acc[j] = fmaf(__uint_as_float(v[j]) * sb.x, sa, acc[j]); acc[j + 1] = fmaf(__uint_as_float(v[j + 1]) * sb.y, sa, acc[j + 1]);
                acc[j + 2] = fmaf(__uint_as_float(v[j + 2]) * sb.z, sa, acc[j + 2]); acc[j + 3] = fmaf(__uint_as_float(v[j + 3]) * sb.w, sa, acc[j + 3]);
            }
        };
        if (n_steps) load(s0);
        uint32_t stage = 0, phase = 1;
        for (uint32_t i = 0; i < n_steps; i++) {
            if (ok) ok = __all_sync(0xffffffffu, mbar_wait(empty + 8 * stage, phase));
            float* const sc = scales + (i & 3) * (kBM + kBN);
            uint8_t* const to = ring + stage * kSgStage;
#pragma unroll
            for (int side = 0; side < 2; side++) {                   // the source's rows, the weights'
                float mx[4];
#pragma unroll
                for (int j = 0; j < 4; j++) { const float4 y = x[4 * side + j]; mx[j] = abs_or_inf(abs_or_inf(abs_or_inf(abs_or_inf(0.0f, y.x), y.y), y.z), y.w); }
#pragma unroll
                for (int o = 8; o > 0; o >>= 1)
#pragma unroll
                    for (int j = 0; j < 4; j++) mx[j] = fmaxf(mx[j], __shfl_xor_sync(0xffffffffu, mx[j], o));
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float4 y = x[4 * side + j];
                    const uint32_t row = r + 32 * j;
                    float scale, inv;
                    split_scale(mx[j], scale, inv);
                    if (c == 0) sc[side * kBM + row] = inv;
                    uint32_t h[2], l[2];
                    split2(y.x * scale, y.y * scale, h[0], l[0]);
                    split2(y.z * scale, y.w * scale, h[1], l[1]);
                    uint8_t* const at = to + side * 2 * kTile + row * 128 + (((c >> 1) ^ (row & 7)) * 16 + (c & 1) * 8);
                    *reinterpret_cast<uint2*>(at) = make_uint2(h[0], h[1]);
                    *reinterpret_cast<uint2*>(at + kTile) = make_uint2(l[0], l[1]);
                }
            }
            if (i + 1 < n_steps) load(s0 + i + 1);                   // in flight while the step before is drained
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(full + 8 * stage);
            if (++stage == kSgStages) { stage = 0; phase ^= 1; }
            if (i) drain(i - 1);
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
            if (m < a.M && n < a.part_rs) *reinterpret_cast<float4*>(p + (size_t)m * a.part_rs + n) = out[rr * 32 + (j ^ (rr & 7))];
        }
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    __syncwarp();
    fence_before();
    __syncthreads();
    if (warp == 16) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(tmem) : "memory");
}

// the shares' sums, bias, activation; four weight rows (pairs: two outputs) per thread
__global__ void __launch_bounds__(256) k_split_finish(const SgArgs a, float* __restrict__ dst, uint32_t dst_rs, const float* __restrict__ bias, SeqAct act, uint32_t pairs) {
    pdl_enter();
    const uint32_t n = 4 * (blockIdx.x * 256 + threadIdx.x), m = blockIdx.y;
    if (n >= a.N) return;
    if (a.rows_from && m / kBM * kBM >= (uint32_t)ctl_word(a.ctl, ZG_CTL_POS) + a.rows_from) return;
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (uint32_t s = 0; s < a.splits; s++) {
        const float4 p = *reinterpret_cast<const float4*>(a.part + ((size_t)s * a.M + m) * a.part_rs + n);
        v.x += p.x; v.y += p.y; v.z += p.z; v.w += p.w;
    }
    float z[4] = {v.x, v.y, v.z, v.w};
    const float* src = a.src + (a.ctl && a.slot_stride ? (size_t)ctl_word(a.ctl, ZG_CTL_SLOT) * a.slot_stride : 0) + (size_t)m * a.src_rs;
#pragma unroll
    for (int j = 0; j < 4; j++)
        if (!(z[j] == z[j]) && n + j < a.N) {                        // not a number: as a plain f32 sum
            float acc = 0.0f;
            for (uint32_t k = 0; k < a.K; k++) acc = fmaf(src[k], a.W[(size_t)(n + j) * a.K + k], acc);
            z[j] = acc;
        }
    float* out = dst + (size_t)m * dst_rs;
    if (pairs) {
#pragma unroll
        for (int j = 0; j < 4; j += 2) if (n + j + 1 < a.N) out[(n + j) / 2] = seq_epilogue(z[j], act.kind, act.p) * z[j + 1];
        return;
    }
#pragma unroll
    for (int j = 0; j < 4; j++)
        if (n + j < a.N) z[j] = seq_epilogue(z[j] + (bias ? bias[n + j] : 0.0f), act, n + j);
    if (n + 4 <= a.N && (reinterpret_cast<uintptr_t>(out + n) & 15) == 0) *reinterpret_cast<float4*>(out + n) = make_float4(z[0], z[1], z[2], z[3]);
    else
        for (int j = 0; j < 4; j++) if (n + j < a.N) out[n + j] = z[j];
}

// shares of K: the fewest rounds of CTAs times steps per CTA, a step of overhead for each round's start and end
uint32_t shares(uint32_t M, uint32_t N, uint32_t K, uint32_t n_sm) {
    const uint32_t tiles = ((M + kBM - 1) / kBM) * ((N + kBN - 1) / kBN), steps = (K + kBK - 1) / kBK;
    uint32_t best = 1, best_cost = ~0u;
    for (uint32_t s = 1; s <= 16 && s <= (steps + 3) / 4; s++) {
        const uint32_t cost = ((tiles * s + n_sm - 1) / n_sm) * ((steps + s - 1) / s + 4) + s / 2;
        if (cost < best_cost) { best_cost = cost; best = s; }
    }
    return best;
}
uint32_t sm_count() {
    static const uint32_t n = [] { int dev = 0, v = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev); return (uint32_t)(v > 0 ? v : 148); }();
    return n;
}
uint32_t up4(uint32_t n) { return (n + 3) / 4 * 4; }

}  // namespace

// rows start at 16-byte boundaries; N counts weight rows
bool zg_split_gemm_usable(const float* w, const float* src, uint32_t M, uint32_t N, uint32_t K, uint32_t src_rs, uint32_t slot_stride) {
    return M > 8 && N >= 32 && K >= 64 && K % 4 == 0 && src_rs % 4 == 0 && slot_stride % 4 == 0 && ((reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(src)) & 15) == 0;
}
size_t zg_split_gemm_scratch_elems(uint32_t M, uint32_t N, uint32_t K) { return (size_t)shares(M, N, K, sm_count()) * M * up4(N); }
bool zg_split_gemm_launch(const float* w, const float* bias, const float* src, float* dst, uint32_t M, uint32_t N, uint32_t K, uint32_t src_rs, uint32_t dst_rs, float* scratch, cudaStream_t st,
                          uint32_t act, float act_p, uint32_t act_lo, uint32_t act_hi, const float* ctl, uint32_t slot_stride, bool pairs, uint32_t rows_from) {
    static const cudaError_t set = cudaFuncSetAttribute(k_split_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSgSmem);
    if (set != cudaSuccess) { zg_set_error("cudaFuncSetAttribute(split gemm) failed: %s", cudaGetErrorString(set)); return false; }
    const SgArgs a = {src, w, scratch, M, N, K, src_rs, up4(N), shares(M, N, K, sm_count()), ctl, slot_stride, rows_from};
    launch_pdl(k_split_gemm, dim3((N + kBN - 1) / kBN, (M + kBM - 1) / kBM, a.splits), dim3(kSgThreads), kSgSmem, st, a);
    ZG_COUNT_LAUNCH();
    launch_pdl(k_split_finish, dim3((N + 1023) / 1024, M), dim3(256), 0, st, a, dst, dst_rs, bias, SeqAct{act, act_p, act_lo, act_hi}, (uint32_t)pairs);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { zg_set_error("split gemm launch failed: %s", cudaGetErrorString(e)); return false; }
    ZG_COUNT_LAUNCH();
    return true;
}
