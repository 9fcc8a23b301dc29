// The layers of a single-token LLaMA program on ONE thread-block cluster of 16 CTAs, for models whose layers are a few MB.
//
// What bounds such a step is the chain of dependent launches: seven per layer, 31 us for the 3.8 MB of a layer of width 576, whose
// bytes pass in 2 - 3 us.  Here a layer is five phases on 16 SMs without a launch between them, and what passes from one to the next
// are vectors in shared memory.  30 layers of width 576 over 512 positions (Q8_0): 975 -> 797 us a token, head and host included, some
// 23 us a layer; other shapes and where the line to the general schedule lies: cluster_pays (backend.cu).  What bounds it now is not
// memory but the walk of the warps through a layer's code: about 2000 instructions a warp, most of them executed once per layer, each
// waiting for the one before it or for its own fetch (some 58 KB of code).  Stamped while a layer took 24 us, 45 000 clocks: attention
// 9000, the four products 1700 - 3500 each, reductions and exchanges between them the rest.
//
//   1  x (residual stream) -> rmsnorm, x inv gamma formed where a record's digits are cut -> q | k | v matvecs, whole columns per CTA
//   2  rope, cache stores, attention: CTA = (KV head, share of the positions), all query heads of the group -> partial states
//   3  merge of the partial states -> o matvec, whole columns -> the owner of a column group adds the residual
//   4  rmsnorm -> gate | up matvecs in pairs -> activation: stays in the CTA
//   5  down matvec over the CTA's own rows of the weight -> partial sums to the owner of the column group, which adds the residual
//
// A producer stores its result straight into the 16 consumers' shared memory (st.async, completion counted by their mbarriers): one
// hop of some 500 clocks where a grid barrier is 1.9 us (decode.cu) and a launch 3 - 5.  The owner of a column group of the residual
// stream sends the group's sum of squares and largest |x gamma| along, so that the consumers need no block-wide reduction: a warp
// goes from the arrival of x to its digit planes without a barrier.  Weights stream through a ring of bulk copies per warp, filled
// by a warp of its own that runs ahead over phases and layers; keys, values and the layer's small operands have such warps as well.
// Records, digit planes and integer products are those of qgemv.cu (see there for the numerics).
//
// Order of stores to an inbox against the reads of what it held before: everything a CTA reads of layer l's inboxes except the
// partial sums of phase 5 is read when it has finished phase 4 and then arrives at every CTA's `go` barrier; nobody sends from phase
// 5 of layer l on before his `go` is complete.  The sums of phase 5 are read by their owners before these send the x of layer l + 1,
// and phase 5 of layer l + 1 follows the arrival of all of that x.
//
// Every DeviceOp's buffer is written (the owners and producers store what they hold).  Every wait is bounded: a CTA that gives up
// counts it, marks the launch, no longer waits and stops before a layer whose operands (addresses among them) have not come; the last
// layer's outputs then come out as NaN.
#include "zg_internal.cuh"
#include "decode_act.cuh"

#include <algorithm>
#include <string.h>

namespace {

constexpr uint32_t kC = kZgClusterCtas;
constexpr uint32_t kW = 16, kT = kW * 32;             // warps that compute
constexpr uint32_t kThreads = kT + 96;                // + weight stream, layer operands, keys and values
__host__ __device__ constexpr uint32_t turn_records(int fmt) { return fmt == ZG_QFMT_I4_F16 ? 4u : 2u; }      // records that a warp takes at a time: a ring slot
__host__ __device__ constexpr uint32_t record_bytes(int fmt) { return fmt == ZG_QFMT_I4_F16 ? 576u : fmt == ZG_QFMT_I8_F32 ? 1152u : 1088u; }
constexpr uint32_t kPlaneRow = 144, kPlaneBytes = 4 * kPlaneRow;
constexpr uint32_t kKvRows = 32;                      // positions of a stage of keys and values
__host__ __device__ constexpr uint32_t max_group(uint32_t dh) { return dh == 128 ? 2u : 4u; }      // query heads of a KV head (three of 128 leave no room for keys and weights)
__host__ __device__ constexpr uint32_t kv_stage_bytes(uint32_t dh) { return (2 * kKvRows * dh + kKvRows) * 4; }      // keys, values, mask
constexpr uint32_t kMaxItems = kZgClusterItems;                    // column groups of a CTA in one phase

enum { kBarA1, kBarQ, kBarT, kBarA2, kBarR, kBarGo, kBarConstFull, kBarConstEmpty = kBarConstFull + 2, kBarKvFull = kBarConstEmpty + 2, kBarKvEmpty = kBarKvFull + 4, kBarFull = kBarKvEmpty + 4 };
// kBarFull: [warp][slot], then the empty barriers the same way

__device__ unsigned int g_timeouts = 0;

__device__ __forceinline__ void imma_s8u8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void imma_u8u8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.relaxed.cta.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Releases the reads before it, its own and (a __syncwarp or a barrier before it) the other lanes': what they read may be overwritten then.  It also waits until the warp's
// stores to global memory are acknowledged, some 25 us of a step of 30 layers; storing later, behind the products, made no difference (788 / 790 us) or cost more (795).
__device__ __forceinline__ void mbar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {      // asks without waiting
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ uint32_t mapa(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
// into another CTA's shared memory, counted there (`at` and `bar` lie in that CTA's window)
__device__ __forceinline__ void push4(uint32_t at, float4 v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(at), "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)),
                 "r"(__float_as_uint(v.z)), "r"(__float_as_uint(v.w)), "r"(bar) : "memory");
}
__device__ __forceinline__ void push1(uint32_t at, float v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(at), "r"(__float_as_uint(v)), "r"(bar) : "memory");
}
__device__ __forceinline__ void arrive_remote(uint32_t bar, uint32_t rank) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(mapa(bar, rank)) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void workers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kT) : "memory"); }
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 r;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(addr));
    return r;
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
    uint32_t r;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(r) : "r"(addr));
    return r;
}
__device__ __forceinline__ uint32_t lds8(uint32_t addr) {
    uint32_t r;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(r) : "r"(addr));
    return r;
}
__device__ __forceinline__ float ldf(uint32_t addr) { return __uint_as_float(lds32(addr)); }
__device__ __forceinline__ float2 ldf2(uint32_t addr) {
    float2 r;
    asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(r.x), "=f"(r.y) : "r"(addr));
    return r;
}
__device__ __forceinline__ float4 ldf4(uint32_t addr) {
    float4 r;
    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w) : "r"(addr));
    return r;
}
template <typename T>
__device__ __forceinline__ T* ldp(uint32_t addr) {
    unsigned long long r;
    asm volatile("ld.shared.u64 %0, [%1];" : "=l"(r) : "r"(addr));
    return reinterpret_cast<T*>(r);
}
__device__ __forceinline__ void stf(uint32_t addr, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }
__device__ __forceinline__ void stf4(uint32_t addr, float4 v) { asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory"); }
__device__ __forceinline__ void sts32(uint32_t addr, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
__device__ __forceinline__ void sts8(uint32_t addr, uint32_t v) { asm volatile("st.shared.u8 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
__device__ __forceinline__ void stg4(float* p, float4 v) { asm volatile("st.global.v4.f32 [%0], {%1,%2,%3,%4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory"); }
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) { return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v))); }   // not negative
__device__ __forceinline__ float abs_or_inf(float a) { a = fabsf(a); return a <= 3.0e38f ? a : INFINITY; }   // NaN counts as infinite
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
__device__ __forceinline__ float4 shfl_add4(float4 v, int o) {
    return make_float4(v.x + __shfl_xor_sync(0xffffffffu, v.x, o), v.y + __shfl_xor_sync(0xffffffffu, v.y, o), v.z + __shfl_xor_sync(0xffffffffu, v.z, o), v.w + __shfl_xor_sync(0xffffffffu, v.w, o));
}
__device__ __forceinline__ float pick(float4 v, uint32_t i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

struct Cta {
    uint8_t* smem;
    uint32_t base, bars;                 // shared-memory addresses
    uint32_t rank, tid, lane, warp;
};
__device__ __forceinline__ uint32_t bar_of(const Cta& c, uint32_t i) { return c.bars + 8 * i; }
// A poll holds the warp for up to 4 us.  Who has polled for some two seconds marks the CTA, and nobody in it waits any more.
constexpr uint32_t kDead = 248, kNoOperands = 252, kPolls = 1u << 19;      // where the mark lies in shared memory, and that of a layer whose operands have not come
__device__ __forceinline__ uint32_t smem_base() {
    extern __shared__ __align__(128) uint8_t smem[];
    return smem_u32(smem);
}
__device__ __forceinline__ bool dead() { return lds32(smem_base() + kDead) != 0; }
__device__ __forceinline__ bool wait_bar(uint32_t bar, uint32_t parity) {      // false: it is not there
    uint32_t polls = 0;
#pragma unroll 1
    while (!mbar_try(bar, parity)) {
        if (++polls == kPolls) sts32(smem_base() + kDead, 1u);
        if (dead()) return false;
    }
    return true;
}

// What a warp's bulk copies have still to bring lands before the warp ends, whatever made it end: their CTA's shared memory must not go before (some 60 ms at most).
__device__ __forceinline__ void settle(uint32_t bar, uint32_t parity) {
#pragma unroll 1
    for (uint32_t polls = 0; polls < (1u << 14) && !mbar_try(bar, parity); polls++) {}
}

// On a barrier that other CTAs complete: what they did before is seen after it.  (Asked for once more at cluster scope, when it is there: an acquire at that scope
// empties the L1 at every poll.)
__device__ __forceinline__ void wait_cluster(uint32_t bar, uint32_t parity) {
    wait_bar(bar, parity);
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%0], %1;\n\t}" ::"r"(bar), "r"(parity) : "memory");
}

// One phase's share of a CTA: `own` column groups of `nk` records each, dealt to the warps as one list of own * nk records.
struct __align__(16) Share { uint32_t own, nk, k0, stride; };      // k0: first record of a column group that is this CTA's; stride: records of a whole column group
__host__ __device__ inline Share share_of(const ZgClusterPlan& P, uint32_t rank, uint32_t ph) {
    Share s;
    const uint32_t nD = P.D >> 5, nQ = P.Dq >> 5, nF = P.F >> 5, lo = rank * nF / kC, hi = (rank + 1) * nF / kC;
    if (ph == 0) { const uint32_t n = nQ + 2 * (P.Dkv >> 5); s.own = (n + kC - 1 - rank) / kC; s.nk = s.stride = nD; s.k0 = 0; }
    else if (ph == 1) { s.own = (nD + kC - 1 - rank) / kC; s.nk = s.stride = nQ; s.k0 = 0; }
    else if (ph == 2) { s.own = 2 * (hi - lo); s.nk = s.stride = nD; s.k0 = 0; }
    else { s.own = hi > lo ? nD : 0; s.nk = hi - lo; s.k0 = lo; s.stride = nF; }
    return s;
}
// where range i of the n records of K ends: those of the warps of the general schedule's matvecs, in each of S splits
__host__ __device__ inline uint32_t range_end(uint32_t n, uint32_t S, uint32_t i) {
    const uint32_t s = i / kZgClusterRanges, ks = s * n / S;
    return ks + (i % kZgClusterRanges + 1) * ((s + 1) * n / S - ks) / kZgClusterRanges;
}
// item i of the phase: its weight, and from bit 8 on its column group there
__host__ __device__ inline uint32_t item_of(const ZgClusterPlan& P, uint32_t rank, uint32_t ph, uint32_t i) {
    if (ph == 0) {
        const uint32_t g = rank + kC * i, nQ = P.Dq >> 5, nK = P.Dkv >> 5;
        return g < nQ ? g << 8 : g < nQ + nK ? ((g - nQ) << 8) | 1 : ((g - nQ - nK) << 8) | 2;
    }
    if (ph == 1) return ((rank + kC * i) << 8) | 3;
    if (ph == 2) return ((rank * (P.F >> 5) / kC + (i >> 1)) << 8) | (4 + (i & 1));
    return (i << 8) | 6;
}

// ── a warp's records of one phase: partial sums of its stretch of every column group that it touches -> part[warp * seg + n][32] ──
// Activations share a scale over the records that lie in one range of the general schedule (a warp's there), so that none is cut on a coarser grid than there: with a scale for
// the whole stretch, seven records instead of two or three, gate and up of width 576 were off by 1.6 times as much beside channels that stand out (a step of 30 layers took 788 us,
// with the ranges 800).
// Addresses in shared memory: x: the K values; gamma: 0, or x * inv * gamma is what is multiplied; top: largest magnitude of 32 values of x (times gamma).
__device__ __noinline__ float true_max(uint32_t x, uint32_t gamma, float inv, uint32_t n) {      // the bound was infinite, the products may not be
    float mx = 0.0f;
#pragma unroll 1
    for (uint32_t j = 0; j < n; j++) {
        float v = ldf(x + 128 * j);
        if (gamma) v = __fmul_rn(__fmul_rn(v, inv), ldf(gamma + 128 * j));
        mx = fmaxf(mx, abs_or_inf(v));
    }
    return warp_max(mx);
}
template <int FMT>
__device__ __forceinline__ void matvec(const Cta& c, const ZgClusterPlan& P, uint2 stretch, uint32_t nk, uint32_t lens, uint32_t x, uint32_t gamma, float inv, uint32_t top, uint32_t smax, uint32_t part,
                                       uint32_t& slot, uint32_t& parity) {
    constexpr bool kI4 = (FMT == ZG_QFMT_I4_F16), kF32 = (FMT == ZG_QFMT_I8_F32);
    constexpr uint32_t QB = kI4 ? 512u : 1024u, SB = kF32 ? 32u : 16u, RB = QB + 4 * SB, G = turn_records(FMT), kSlotBytes = G * RB;
    static_assert(RB == record_bytes(FMT), "record");
    const uint32_t lane = c.lane, warp = c.warp, gq = lane >> 2, t = lane & 3;
    lens += stretch.x >> 16;
    uint32_t left = stretch.x & 0xffffu, item = stretch.y & 0xffffu, k = stretch.y >> 16;
    uint32_t out = part + warp * P.seg * 128 + ((t >> 1) * 16 + gq + 8 * (t & 1)) * 4;
    if (left == 0) {         // fewer records than warps: the sum over the warps of an item passes this one
        stf(out, 0.0f);
        return;
    }
    const uint32_t planes = c.base + P.o_planes + warp * kPlaneBytes, brow = planes + (gq & 3) * 32 + 4 * t;
    const uint32_t sc_off = QB + (kF32 ? 4u : 2u) * (8 * ((lane & 15) >> 2) + 4 * (lane >> 4) + (lane & 3));
    const uint32_t ring = c.base + P.o_ring + warp * P.ring_slots * kSlotBytes, full = bar_of(c, kBarFull + warp * P.ring_slots), empty = full + 8 * kW * P.ring_slots;
    float sum = 0.0f;
#pragma unroll 1
    while (left) {
        const uint32_t n = lds8(lens++);
        float mx = 0.0f;
#pragma unroll 1
        for (uint32_t j = lane; j < n; j += 32) mx = fmaxf(mx, ldf(top + (k + j) * 4));
        const float sm = ldf(smax + item * 4);
        mx = warp_max(mx);
        uint32_t xk = x + (k * 32 + lane) * 4, gk = gamma + (k * 32 + lane) * 4;
        if (gamma) mx *= inv;
        if (!(mx <= 3.0e38f)) mx = true_max(xk, gamma ? gk : 0, inv, n);
        const float f = (mx <= 3.0e38f && mx >= 1.0e-30f) ? (0.499f / mx) * (1.0f / sm) : 0.0f;
        int acc[2][4] = {};
        uint32_t dsum = 0;
        // G records a turn.  Those past the end have 1.5 for every digit's value: what they add to the sums of digits the sum of weights takes away again.
#pragma unroll 1
        for (uint32_t r0 = 0; r0 < n; r0 += G, xk += G * 128, gk += G * 128) {
            const uint32_t at = ring + slot * kSlotBytes;
            float v[G];
#pragma unroll
            for (uint32_t r = 0; r < G; r++) v[r] = ldf(xk + 128 * r);
            if (gamma) {
#pragma unroll
                for (uint32_t r = 0; r < G; r++) v[r] = __fmul_rn(__fmul_rn(v[r], inv), ldf(gk + 128 * r));
            }
            wait_bar(full + 8 * slot, parity);
            // digit planes: lane = row of the weight; the low three bytes are base-256 digits
#pragma unroll
            for (uint32_t r = 0; r < G; r++) {
                float sc;
                if constexpr (kF32) {
                    sc = ldf(at + sc_off + r * RB);
                } else {
                    unsigned short h;
                    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(h) : "r"(at + sc_off + r * RB));
                    sc = __half2float(__ushort_as_half(h));
                }
                const float Fv = fmaf(sc, v[r] * f, 1.5f);
                const uint32_t F = __float_as_uint(r == 0 || r0 + r < n ? Fv : 1.5f), pa = planes + lane + r * kPlaneRow;
                sts8(pa, F);
                sts8(pa + 32, F >> 8);
                sts8(pa + 64, F >> 16);
            }
            __syncwarp();
#pragma unroll
            for (uint32_t r = 0; r < G; r++) {
                const uint32_t qa = at + lane * 16 + r * RB, b0 = lds32(brow + r * kPlaneRow), b1 = lds32(brow + r * kPlaneRow + 16);
                if constexpr (!kI4) {
                    const uint4 q0 = lds128(qa), q1 = lds128(qa + 512);
                    imma_s8u8(acc[0], q0.x, q0.y, q0.z, q0.w, b0, b1);
                    imma_s8u8(acc[1], q1.x, q1.y, q1.z, q1.w, b0, b1);
                } else {
                    const uint4 q0 = lds128(qa);
                    dsum = __dp4a(b0, 0x01010101u, __dp4a(b1, 0x01010101u, dsum));
                    imma_u8u8(acc[0], q0.x, q0.x & 0x0F0F0F0Fu, q0.y, q0.y & 0x0F0F0F0Fu, b0, b1);
                    imma_u8u8(acc[1], q0.z, q0.z & 0x0F0F0F0Fu, q0.w, q0.w & 0x0F0F0F0Fu, b0, b1);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty + 8 * slot);
            if (++slot == P.ring_slots) { slot = 0; parity ^= 1; }
        }
        // Integer sums -> the warp's partial of the column group, one column a lane.  The product's columns are the three digits and the plane of ones, twice: lanes t = 0, 1
        // of a row share those of the first 16 columns, t = 2, 3 those of the others; the even one takes row gq, the odd one row gq + 8.
        const bool second = t & 2, odd = t & 1;
        int p0 = second ? acc[1][0] : acc[0][0], p1 = second ? acc[1][1] : acc[0][1], q0 = second ? acc[1][2] : acc[0][2], q1 = second ? acc[1][3] : acc[0][3];
        long long dS = 0;
        if constexpr (kI4) {      // rows gq: both nibbles, rows gq + 8: the low ones
            const int hi0 = (p0 - q0) >> 4, hi1 = (p1 - q1) >> 4;
            p0 = q0; p1 = q1; q0 = hi0; q1 = hi1;
            uint32_t ds = dsum;
            ds += __shfl_xor_sync(0xffffffffu, ds, 1);
            ds += __shfl_xor_sync(0xffffffffu, ds, 2);
            const uint32_t D0 = __shfl_sync(0xffffffffu, ds, 0), D1 = __shfl_sync(0xffffffffu, ds, 4), D2 = __shfl_sync(0xffffffffu, ds, 8);
            dS = (long long)D0 + ((long long)D1 << 8) + ((long long)D2 << 16);
        }
        const int r0 = __shfl_xor_sync(0xffffffffu, odd ? p0 : q0, 1), r1 = __shfl_xor_sync(0xffffffffu, odd ? p1 : q1, 1);
        const int d0 = odd ? r0 : p0, d1 = odd ? r1 : p1, d2 = odd ? q0 : r0, ones = odd ? q1 : r1;
        long long T = (long long)d0 + (long long)d1 * 256 + (long long)d2 * 65536;
        if constexpr (kI4) T += -8 * dS - 12582912LL * (ones - 8LL * (long long)((n + G - 1) / G * G * ZG_KR));
        else T -= 12582912LL * ones;
        const float esc = (mx <= 3.0e38f) ? ((mx >= 1.0e-30f) ? (mx * (2.004008016f * 1.1920928955078125e-07f)) * sm : 0.0f) : __int_as_float(0x7fc00000);
        sum = fmaf(__ll2float_rn(T), esc, sum);
        left -= n; k += n;
        if (k == nk || left == 0) {
            stf(out, sum);
            out += 128;
            sum = 0.0f; k = 0; item++;
        }
    }
}
// sum of an item's partials: columns c4 .. c4 + 3, by the four dg of a warp together; entry: first and last warp that hold some, and which of its pieces the first one's is
__device__ __forceinline__ float4 part_sum(uint32_t part, uint32_t entry, uint32_t seg, uint32_t c4, uint32_t dg) {
    const uint32_t lo = entry & 255u, hi = (entry >> 8) & 255u, at = part + c4 * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    uint32_t w = lo + dg;
    if (w <= hi) v = ldf4(at + (w * seg + (dg == 0 ? entry >> 16 : 0)) * 128);
#pragma unroll 1
    for (w += 4; w - dg <= hi; w += 4)
        if (w <= hi) v = add4(v, ldf4(at + w * seg * 128));
    return shfl_add4(shfl_add4(v, 8), 16);
}

__device__ __forceinline__ float inv_rms(uint32_t ss, uint32_t n, uint32_t lane, float D, float eps) {
    float v = lane < n ? ldf(ss + lane * 4) : 0.0f;
#pragma unroll 1
    for (uint32_t i = lane + 32; i < n; i += 32) v += ldf(ss + i * 4);
    return 1.0f / sqrtf(warp_sum(v) / D + eps);
}

// ── attention of the CTA's share of the positions, all query heads of its KV head ──
__device__ __forceinline__ uint32_t head_lane(uint32_t h) { return ((h & 1) << 1) | (h >> 1); }      // which of a position's eight lanes has head h's score
template <int NI, int GS>
__device__ __noinline__ void attention_share(uint32_t kv, uint32_t bars, uint32_t stages_log2, uint32_t sq, uint32_t state, uint32_t at_, uint32_t t_at, uint32_t t_stride, uint32_t base,
                                             float qk_scale) {
    constexpr uint32_t dh = NI * 32;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane >> 3, sg = lane & 7, half = warp >> 3, lo = lds32(at_ + 24), len = lds32(at_ + 28), s_new = lds32(at_ + 16);
    const uint32_t sk = sq + GS * dh * 4, sv = sk + dh * 4, head = ((sg & 1) << 1) | ((sg >> 1) & 1);
    const uint32_t seqh = head < GS ? lds32(at_ + head * 4) : 0;
    float m = -INFINITY, l = 0.0f, acc[GS][NI];
#pragma unroll
    for (int h = 0; h < GS; h++)
#pragma unroll
        for (int i = 0; i < NI; i++) acc[h][i] = 0.0f;
    const uint32_t stages = (len + kKvRows - 1) / kKvRows;
#pragma unroll 1
    for (uint32_t at = half; at < stages; at += 2) {
        const uint32_t cum = base + at, st = cum & ((1u << stages_log2) - 1), row0 = (warp & 7) * 4, p0 = at * kKvRows + row0;
        wait_bar(bars + 8 * (kBarKvFull + st), (cum >> stages_log2) & 1);
        if (p0 < len) {
            const uint32_t cnt = min(4u, len - p0), r = min(sub, cnt - 1), s = lo + p0 + r, stage = kv + st * kv_stage_bytes(dh), K = stage + row0 * dh * 4, V = K + kKvRows * dh * 4;
            const uint32_t kr = (s == s_new ? sk : K + r * dh * 4) + sg * 16;
            const float mask_add = ldf(stage + (2 * kKvRows * dh + row0 + r) * 4);
            float dot[4] = {};
#pragma unroll
            for (int i = 0; i < NI; i++) {
                const float4 a = ldf4(kr + 128 * i);
#pragma unroll
                for (int h = 0; h < GS; h++) {
                    const float4 q = ldf4(sq + h * dh * 4 + sg * 16 + 128 * i);
                    dot[h] = fmaf(q.x, a.x, fmaf(q.y, a.y, fmaf(q.z, a.z, fmaf(q.w, a.w, dot[h]))));
                }
            }
            // sums over the eight lanes, each of which is left with one head's
            const bool b0 = sg & 1, b1 = sg & 2;
            float d0 = b0 ? dot[2] : dot[0], d1 = b0 ? dot[3] : dot[1];
            if (GS > 2) d0 += __shfl_xor_sync(0xffffffffu, b0 ? dot[0] : dot[2], 1); else d0 = dot[0] + __shfl_xor_sync(0xffffffffu, dot[0], 1);
            if (GS > 1) d1 = GS > 2 ? d1 + __shfl_xor_sync(0xffffffffu, b0 ? dot[1] : dot[3], 1) : dot[1] + __shfl_xor_sync(0xffffffffu, dot[1], 1);
            float score = (b1 ? d1 : d0) + __shfl_xor_sync(0xffffffffu, b1 ? d0 : d1, 2);
            score += __shfl_xor_sync(0xffffffffu, score, 4);
            score = score * qk_scale + mask_add;
            if (!(sub < cnt && s < seqh && isfinite(mask_add) && isfinite(score))) score = -INFINITY;
            float nm = fmaxf(score, __shfl_xor_sync(0xffffffffu, score, 8));
            nm = fmaxf(m, fmaxf(nm, __shfl_xor_sync(0xffffffffu, nm, 16)));
            const float alpha = m == -INFINITY ? 0.0f : expf(m - nm), w = score == -INFINITY ? 0.0f : expf(score - nm);
            l = fmaf(l, alpha, w);            // of the lane's own positions
            m = nm;
#pragma unroll
            for (int h = 0; h < GS; h++) {
                const float ah = __shfl_sync(0xffffffffu, alpha, head_lane(h));
#pragma unroll
                for (int i = 0; i < NI; i++) acc[h][i] *= ah;
            }
#pragma unroll
            for (uint32_t j = 0; j < 4; j++) {
                if (j < cnt) {
                    const uint32_t vr = (lo + p0 + j == s_new ? sv : V + j * dh * 4) + lane * 4;
                    float vv[NI];
#pragma unroll
                    for (int i = 0; i < NI; i++) vv[i] = ldf(vr + 128 * i);
#pragma unroll
                    for (int h = 0; h < GS; h++) {
                        const float wj = __shfl_sync(0xffffffffu, w, j * 8 + head_lane(h));
                        if (wj != 0.0f) {             // a position that does not count may hold anything
#pragma unroll
                            for (int i = 0; i < NI; i++) acc[h][i] = fmaf(wj, vv[i], acc[h][i]);
                        }
                    }
                }
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bars + 8 * (kBarKvEmpty + st));
    }
    // the warps' maxima, then their sums against the common one
    if (sub == 0 && sg < 4 && head < GS) stf(state + (head * kW + warp) * 4, m);
    l += __shfl_xor_sync(0xffffffffu, l, 8);
    l += __shfl_xor_sync(0xffffffffu, l, 16);
    workers_sync();
    float top[4];
#pragma unroll
    for (int h = 0; h < GS; h += 2) {
        float v = h + (lane >> 4) < GS ? ldf(state + ((h + (lane >> 4)) * kW + (lane & 15)) * 4) : -INFINITY;
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
        top[h] = __shfl_sync(0xffffffffu, v, 0);
        top[h + 1] = __shfl_sync(0xffffffffu, v, 16);
    }
    const float mine = head == 0 ? top[0] : head == 1 ? top[1] : GS > 2 ? (head == 2 ? top[2] : top[3]) : top[0];
    const float scale = m == -INFINITY ? 0.0f : expf(m - mine);
    const uint32_t rows = state + GS * kW * 4;             // [head][warp][dh + 4]: the sums, their weight
#pragma unroll
    for (int h = 0; h < GS; h++) {
        const float sh = __shfl_sync(0xffffffffu, scale, head_lane(h)), lh = __shfl_sync(0xffffffffu, l, head_lane(h)) * sh;
        const uint32_t row = rows + (h * kW + warp) * (dh + 4) * 4;
#pragma unroll
        for (int i = 0; i < NI; i++) stf(row + (lane + 32 * i) * 4, acc[h][i] * sh);
        if (lane == 0) stf4(row + dh * 4, make_float4(lh, top[h], 0.f, 0.f));
    }
    workers_sync();
    // four elements an eighth of a warp, two warps' sums a lane, sent to two CTAs a lane
    constexpr uint32_t Q = dh / 4 + 1;
    const uint32_t j = lane & 7;
    uint32_t w0, w1, bar0;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(w0) : "r"(t_at), "r"(j));
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(w1) : "r"(t_at), "r"(j + 8));
    bar0 = bars + 8 * kBarT - t_at;
#pragma unroll 1
    for (uint32_t q = warp * 4 + (lane >> 3); q < ((GS * Q + 3) & ~3u); q += 4 * kW) {
        const uint32_t h = min(q / Q, (uint32_t)GS - 1), e = q - h * Q;
        const uint32_t row = rows + ((h * kW + j) * (dh + 4) + e * 4) * 4;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
        if (q < GS * Q) a = add4(ldf4(row), ldf4(row + 8 * (dh + 4) * 4));
        a = shfl_add4(shfl_add4(shfl_add4(a, 1), 2), 4);
        if (e == dh / 4) a.y = ldf(row + 4);      // the common maximum, as every warp wrote it
        if (q < GS * Q) {
            push4(w0 + (h * t_stride + e * 4) * 4, a, w0 + bar0);
            push4(w1 + (h * t_stride + e * 4) * 4, a, w1 + bar0);
        }
    }
}

// this CTA's share of a layer's positions
__device__ __forceinline__ void kv_share(const ZgClusterPlan& P, uint32_t split, uint32_t seq_max, uint32_t& lo, uint32_t& len) {
    const uint32_t chunk = ((seq_max + P.splits - 1) / P.splits + 3) & ~3u;
    lo = split * chunk;
    len = seq_max > lo ? min(chunk, seq_max - lo) : 0;
}

// One lane per worker warp walks that warp's list of copies {weight, offset, bytes}, layer after layer (copy_list).
__device__ __noinline__ void weight_stream(const ZgClusterPlan* plan) {
    const ZgClusterPlan& P = *plan;
    const uint32_t base = smem_base(), lane = threadIdx.x & 31, w = min(lane, kW - 1), ring = base + P.o_ring + w * P.ring_slots * P.slot_bytes;
    const uint32_t full = base + P.o_bars + 8 * (kBarFull + w * P.ring_slots), list = base + P.o_list + w * P.list_max * 8, n = lds32(base + P.o_list + (kW * P.list_max * 2 + w) * 4);
    uint32_t slot = 0, wrapped = 0, idle = 0, i = 0, ptrs = base + P.o_ptrs, last = ptrs + (P.n_layers - 1) * 56;
    bool left = lane < kW && n;
#pragma unroll 1
    while (__any_sync(0xffffffffu, left)) {       // every lane asks in turn: none waits for another's slot
        const bool go = left && (!wrapped || mbar_test(full + 8 * (kW * P.ring_slots + slot), (wrapped - 1) & 1));
        if (go) {
            const uint32_t e = lds32(list + i * 8), bytes = e >> 8;
            const uint8_t* src = ldp<const uint8_t>(ptrs + (e & 255u)) + lds32(list + i * 8 + 4);
            mbar_expect_tx(full + 8 * slot, bytes);
            bulk_g2s(ring + slot * P.slot_bytes, src, bytes, full + 8 * slot);
            if (++slot == P.ring_slots) { slot = 0; wrapped++; }
            if (++i == n) { i = 0; left = ptrs != last; ptrs += 56; }
        }
        if (__any_sync(0xffffffffu, go)) { idle = 0; continue; }
        if (idle == 0) asm volatile("griddepcontrol.wait;" ::: "memory");      // no slot comes free before the predecessor has completed, however long that takes: no bounded wait before
        __nanosleep(100);
        if (++idle > (1u << 23) || dead()) break;      // a second and more
    }
#pragma unroll 1
    for (uint32_t s = 0; s < P.ring_slots; s++) {
        const uint32_t fills = wrapped + (s < slot);
        if (lane < kW && fills) settle(full + 8 * s, (fills - 1) & 1);
    }
}
// The list of a warp's copies in one layer: entry {8 * weight | bytes << 8, offset}; counts behind the lists.  And of its stretches: records and first of their ranges' lengths,
// first column group and record.  By one lane per warp, before the start.
template <int FMT>
__device__ __noinline__ void copy_list(const ZgClusterPlan* plan, uint32_t w) {
    constexpr uint32_t RB = record_bytes(FMT), G = turn_records(FMT);
    extern __shared__ __align__(128) uint8_t smem[];
    const ZgClusterPlan& P = *plan;
    uint32_t* lists = reinterpret_cast<uint32_t*>(smem + P.o_list);
    const Share* shares = reinterpret_cast<const Share*>(smem + P.o_table);
    const uint32_t* items = reinterpret_cast<const uint32_t*>(shares + 4);
    const uint32_t* ranges = reinterpret_cast<const uint32_t*>(smem + P.o_ranges);
    uint8_t* lens = smem + P.o_lens;
    uint32_t n = 0, n_ranges = 0;
#pragma unroll 1
    for (uint32_t ph = 0; ph < 4; ph++) {
        const Share s = shares[ph];
        const uint32_t R = s.own * s.nk, end = ((w + 1) * R) / kW;
        uint32_t pos = (w * R) / kW, item = s.nk ? pos / s.nk : 0, k = pos - item * s.nk;
        const uint32_t stretches = P.o_table + 4 * sizeof(Share) + 8 * kMaxItems * 4 + (ph * kW + w) * 8;
        reinterpret_cast<uint32_t*>(smem + stretches)[0] = (end - pos) | (n_ranges << 16);
        reinterpret_cast<uint32_t*>(smem + stretches)[1] = item | (k << 16);
        uint32_t range = 0;      // left of the records that share a scale
#pragma unroll 1
        while (pos < end) {
            if (!range) {
                const uint32_t at = s.k0 + k;
                uint32_t word = at >> 5, ends = ranges[ph * P.range_words + word] & (~0u << (at & 31));
                while (!ends) ends = ranges[ph * P.range_words + ++word];
                range = min(word * 32 + __ffs(ends) - at, min(s.nk - k, end - pos));
                lens[w * P.list_max + n_ranges++] = (uint8_t)range;
            }
            const uint32_t it = items[ph * kMaxItems + item], m = min(G, range);
            range -= m;
            lists[(w * P.list_max + n) * 2] = (it & 255u) * 8 | (m * RB) << 8;
            lists[(w * P.list_max + n) * 2 + 1] = ((it >> 8) * s.stride + s.k0 + k) * RB;
            n++; pos += m; k += m;
            if (k == s.nk) { k = 0; item++; }
        }
    }
    lists[kW * P.list_max * 2 + w] = n;
}

// keys, values and mask of the CTA's positions, as far ahead as there are stages and the layers' operands are there
__device__ __noinline__ void kv_stream(const ZgClusterPlan* plan, uint32_t rank) {
    const ZgClusterPlan& P = *plan;
    const uint32_t lane = threadIdx.x & 31, g = rank / P.splits, base = smem_base(), bars = base + P.o_bars;
    if (g >= P.n_kv) return;
    const uint32_t row = P.dh * 4, stage = kv_stage_bytes(P.dh), lg = P.kv_stages == 4 ? 2 : 1;
    uint32_t cum = 0;
#pragma unroll 1
    for (uint32_t l = 0; l < P.n_layers; l++) {
        const uint32_t area = base + P.o_const + (l & 1) * P.const_bytes, kv = area + (uint32_t)sizeof(ZgClusterLayer) + P.n_heads * (uint32_t)sizeof(ZgClusterHead) + g * (uint32_t)sizeof(ZgClusterKv);
        if (!__all_sync(0xffffffffu, wait_bar(bars + 8 * (kBarConstFull + (l & 1)), (l >> 1) & 1))) break;      // (what would be read there are addresses)
        const uint32_t at = area + P.const_bytes - 48, lo = lds32(at + 24), len = lds32(at + 28), mask_rs = lds32(area + (uint32_t)offsetof(ZgClusterLayer, mask_rs));
        const uint8_t* K = ldp<const uint8_t>(area + (uint32_t)offsetof(ZgClusterLayer, k_cache)) + (size_t)(lds32(kv + (uint32_t)offsetof(ZgClusterKv, k_off)) + lo * P.dh) * 4;
        const uint8_t* V = ldp<const uint8_t>(area + (uint32_t)offsetof(ZgClusterLayer, v_cache)) + (size_t)(lds32(kv + (uint32_t)offsetof(ZgClusterKv, v_off)) + lo * P.dh) * 4;
        const float* mask = lds32(area + (uint32_t)offsetof(ZgClusterLayer, has_mask)) ? ldp<const float>(area + (uint32_t)offsetof(ZgClusterLayer, mask)) + lds32(area + (uint32_t)offsetof(ZgClusterLayer, mask_off)) : nullptr;
        __syncwarp();
        if (lane == 0) mbar_arrive(bars + 8 * (kBarConstEmpty + (l & 1)));
#pragma unroll 1
        for (uint32_t p = 0; p < len; p += kKvRows, cum++) {
            const uint32_t st = cum & (P.kv_stages - 1), turn = cum >> lg, bytes = min(kKvRows, len - p) * row;
            const float m = mask ? __ldcg(mask + (size_t)(lo + min(p + lane, len - 1)) * mask_rs) : 0.0f;
            if (turn) wait_bar(bars + 8 * (kBarKvEmpty + st), (turn - 1) & 1);
            if (dead()) { l = P.n_layers; break; }
            const uint32_t dst = base + P.o_kv + st * stage, bar = bars + 8 * (kBarKvFull + st);
            stf(dst + 2 * kKvRows * row + lane * 4, m);
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");      // releases the mask
            if (lane == 0) {
                mbar_expect_tx(bar, 2 * bytes);
                bulk_g2s(dst, K + (size_t)p * row, bytes, bar);
                bulk_g2s(dst + kKvRows * row, V + (size_t)p * row, bytes, bar);
            }
        }
    }
#pragma unroll 1
    for (uint32_t st = 0; st < min(cum, P.kv_stages); st++) settle(bars + 8 * (kBarKvFull + st), ((cum - 1 - st) >> lg) & 1);
}

// The layer's small operands, one layer ahead: [block][gamma1][gamma2][cos | sin][scale ceilings of the CTA's column groups][positions: those of the heads, the new one
// (as its rows are numbered), where its key and value go, the first and the number of the CTA's]
__device__ __noinline__ void const_stream(const ZgClusterPlan* plan, uint32_t rank) {
    const ZgClusterPlan& P = *plan;
    const uint32_t lane = threadIdx.x & 31, g = rank / P.splits, split = rank - g * P.splits, base = smem_base(), bars = base + P.o_bars;
    const ZgClusterLayer* ly = reinterpret_cast<const ZgClusterLayer*>(P.blocks);
    const float* smax = P.smax + (size_t)rank * 4 * kMaxItems;
    uint32_t l = 0;
#pragma unroll 1
    for (; l < P.n_layers; l++) {
        if (l >= 2) wait_bar(bars + 8 * (kBarConstEmpty + (l & 1)), ((l >> 1) - 1) & 1);
        if (dead()) break;
        const uint32_t area = base + P.o_const + (l & 1) * P.const_bytes, at = area + P.const_bytes - 48, bar = bars + 8 * (kBarConstFull + (l & 1));
        if (lane < 5) {
            const void* src = lane == 0 ? (const void*)ly : lane == 1 ? (const void*)ly->gamma[0] : lane == 2 ? (const void*)ly->gamma[1] : lane == 3 ? (const void*)ly->cs : (const void*)smax;
            const uint32_t bytes = lane == 0 ? P.blk_bytes : lane < 3 ? P.D * 4 : lane == 3 ? P.dh * 4 : 16 * kMaxItems;
            const uint32_t dst = area + (lane == 0 ? 0 : P.blk_bytes + (lane - 1) * P.D * 4 - (lane == 4 ? (P.D - P.dh) * 4 : 0));
            asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
            bulk_g2s(dst, src, bytes, bar);
        }
        if (g < P.n_kv) {
            const ZgClusterHead* hd = reinterpret_cast<const ZgClusterHead*>(ly + 1);
            const ZgClusterKv* kv = reinterpret_cast<const ZgClusterKv*>(hd + P.n_heads) + g;
            const uint32_t mine = __ldcg(P.dyn + (lane < P.gs ? hd[g * P.gs + lane].dyn : lane == 8 ? kv->v_dyn : lane < 8 ? kv->k_dyn : hd[g * P.gs].dyn));
            const uint32_t seq = __reduce_max_sync(0xffffffffu, lane < P.gs ? mine : 0);
            uint32_t lo, len;
            kv_share(P, split, seq, lo, len);
            const uint32_t v = lane < 4 || lane == 8 || lane == 5 ? mine : lane == 4 ? (mine - kv->k_off) >> P.dh_log2 : lane == 6 ? lo : len;
            if (lane < 9) asm volatile("st.shared.u32 [%0], %1;" ::"r"(at + lane * 4), "r"(v) : "memory");
        }
        __syncwarp();
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");      // releases what the lanes have stored
        ly = reinterpret_cast<const ZgClusterLayer*>(reinterpret_cast<const uint8_t*>(ly) + P.blk_bytes);
        smax += kC * 4 * kMaxItems;
    }
    if (l > 1) settle(bars + 8 * (kBarConstFull + (l & 1)), ((l - 2) >> 1) & 1);
    if (l) settle(bars + 8 * (kBarConstFull + ((l - 1) & 1)), ((l - 1) >> 1) & 1);
}

template <int NI>
__device__ __forceinline__ void attend(uint32_t gs, uint32_t kv, uint32_t bars, uint32_t lg, uint32_t sq, uint32_t state, uint32_t at, uint32_t t_at, uint32_t t_stride, uint32_t base,
                                       float scale) {
    if (gs == 1) attention_share<NI, 1>(kv, bars, lg, sq, state, at, t_at, t_stride, base, scale);
    else if (gs == 2) attention_share<NI, 2>(kv, bars, lg, sq, state, at, t_at, t_stride, base, scale);
    else if constexpr (max_group(32 * NI) > 2) {
        if (gs == 3) attention_share<NI, 3>(kv, bars, lg, sq, state, at, t_at, t_stride, base, scale);
        else attention_share<NI, 4>(kv, bars, lg, sq, state, at, t_at, t_stride, base, scale);
    }
}
#define LY(field) (area + (uint32_t)offsetof(ZgClusterLayer, field))

// What bounds a layer is the length of this function: sixteen warps walk through it once per layer, mostly one instruction after the other.  Hence the four matvec phases
// are one loop (with a copy of each per phase a layer took 28 us), reductions are spread over the lanes that are there, and nothing is computed that another CTA can send.
template <int FMT>
__device__ __forceinline__ void workers(const Cta& c, const ZgClusterPlan& P) {
    const uint32_t lane = c.lane, warp = c.warp, tid = c.tid, rank = c.rank, c4 = (lane & 7) * 4, dg = lane >> 3;
    const uint32_t nD = P.D >> 5, nQ = P.Dq >> 5, dh = P.dh, gs = P.gs;
    const uint32_t g = rank / P.splits, split = rank - g * P.splits;
    const bool attends = g < P.n_kv;
    const uint32_t q_in = c.base + P.o_q, t_in = c.base + P.o_t, ao = c.base + P.o_ao, ao_top = ao + P.Dq * 4, hid = c.base + P.o_hid, hid_top = hid + P.hid_max * 4, sq = c.base + P.o_sq;
    const uint32_t shares = c.base + P.o_table, items = shares + 4 * sizeof(Share), table = items + 16 * kMaxItems, stretches = table + 16 * kMaxItems;
    const uint32_t ownD = (nD + kC - 1 - rank) / kC, own_i = (rank + kC * warp) * 32 + c4;      // the warp's own column group of the residual stream, if warp < ownD
    const uint32_t tx_a = (P.D + 2 * nD) * 4, pair0 = rank * (P.F >> 5) / kC;
    uint32_t away[4];                    // what takes an address here to the windows of the four CTAs that this lane sends to
#pragma unroll
    for (uint32_t u = 0; u < 4; u++) away[u] = mapa(c.base, dg * 4 + u) - c.base;
    uint32_t slot = 0, parity = 0, kv_base = 0;
    float4 xown = make_float4(0.f, 0.f, 0.f, 0.f);

    asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll 1
    for (uint32_t l = 0; l < P.n_layers; l++) {
        const uint32_t area = c.base + P.o_const + (l & 1) * P.const_bytes, heads = area + (uint32_t)sizeof(ZgClusterLayer), gammas = area + P.blk_bytes;
        const uint32_t cs = gammas + 8 * P.D, smax = cs + dh * 4, at = smax + 16 * kMaxItems;
        // a layer without its operands has no addresses either: nothing is stored there (set before a barrier, asked for behind it: the same to all)
        if (!wait_bar(bar_of(c, kBarConstFull + (l & 1)), (l >> 1) & 1)) sts32(c.base + kNoOperands, 1u);
        if (l == 0) {      // the program's input: every CTA takes all of it
            workers_sync();
            if (lds32(c.base + kNoOperands)) return;
            const uint32_t a1 = c.base + P.o_a1;
            const float* x_in = ldp<const float>(LY(x_in));
#pragma unroll 1
            for (uint32_t i = warp; i < nD; i += kW) {
                const float v = __ldcg(x_in + i * 32 + lane), ss = warp_sum(v * v), mx = warp_max(abs_or_inf(v * ldf(gammas + (i * 32 + lane) * 4)));
                stf(a1 + (i * 32 + lane) * 4, v);
                if (lane == 0) { stf(a1 + (P.D + i) * 4, ss); stf(a1 + (P.D + nD + i) * 4, mx); }
            }
            workers_sync();
            if (warp < ownD) xown = ldf4(a1 + own_i * 4);
        }
#pragma unroll 1
        for (uint32_t ph = 0; ph < 4; ph++) {
            const uint32_t own = lds32(shares + ph * (uint32_t)sizeof(Share)), nk = lds32(shares + ph * (uint32_t)sizeof(Share) + 4);
            uint32_t x = hid, gamma = 0, top = hid_top;
            float inv = 1.0f, ext = 0.0f;
            const float* sec = nullptr;
            if ((ph & 1) == 0) {
                // ── x has arrived: rmsnorm ──
                if (ph == 2) {      // the activation's constant operand, before the wait
                    const int first = (int)lds32(LY(first_ext));
                    if (first >= 0) {
                        sec = ldp<const float>(LY(steps) + first * (uint32_t)sizeof(ZgDecStep) + (uint32_t)offsetof(ZgDecStep, sec)) + pair0 * 32 + c4 + dg;
                        if (2 * warp < own) ext = __ldcg(sec + warp * 32);
                    }
                }
                const uint32_t bar = bar_of(c, ph ? kBarA2 : kBarA1);
                if (ph | l) {
                    wait_cluster(bar, (ph ? l : l - 1) & 1);
                    if (tid == 0) mbar_expect_tx(bar, tx_a);
                }
                x = c.base + (ph ? P.o_a2 : P.o_a1); top = x + (P.D + nD) * 4; gamma = gammas + (ph ? P.D * 4 : 0);
                inv = inv_rms(x + P.D * 4, nD, lane, (float)P.D, ldf(LY(eps) + ph * 2));
            } else if (ph == 1) {
                // ── rope, cache, attention over the CTA's positions ──
                const uint32_t kv = heads + P.n_heads * (uint32_t)sizeof(ZgClusterHead) + g * (uint32_t)sizeof(ZgClusterKv);
                wait_cluster(bar_of(c, kBarQ), l & 1);
                if (tid == 0) mbar_expect_tx(bar_of(c, kBarQ), (P.Dq + 2 * P.Dkv) * 4);
                if (attends) {
                    const uint32_t hd2 = dh >> 1;
#pragma unroll 1
                    for (uint32_t e = tid; e < (gs + 2) * dh; e += kT) {
                        const uint32_t h = e >> P.dh_log2, r = e & (dh - 1), src = q_in + (h < gs ? (g * gs + h) * dh : P.Dq + (h == gs ? 0 : P.Dkv) + g * dh) * 4;
                        float v = ldf(src + r * 4);
                        if (h <= gs) {            // separate roundings like the reference (reference.zig:474-475)
                            const float cc = ldf(cs + (r & (hd2 - 1)) * 4), t = __fmul_rn(ldf(src + (r ^ hd2) * 4), ldf(cs + (hd2 + (r & (hd2 - 1))) * 4));
                            v = __fadd_rn(__fmul_rn(v, cc), r < hd2 ? -t : t);
                        }
                        stf(sq + e * 4, v);
                        if (split == 0) {
                            if (h <= gs) ldp<float>(h < gs ? heads + (g * gs + h) * (uint32_t)sizeof(ZgClusterHead) : kv)[r] = v;      // q_rot, k_rot: the first fields
                            if (h >= gs) (ldp<float>(h == gs ? LY(k_cache) : LY(v_cache)) + lds32(at + (h == gs ? 20 : 32)))[r] = v;
                        }
                    }
                    workers_sync();
                    const uint32_t lg = P.kv_stages == 4 ? 2 : 1, t_at = t_in + (g * gs * P.splits + split) * (dh + 4) * 4, t_stride = P.splits * (dh + 4);
                    if (dh == 64) attend<2>(gs, c.base + P.o_kv, c.bars, lg, sq, c.base + P.o_state, at, t_at, t_stride, kv_base, ldf(LY(scale)));
                    else if (dh == 128) attend<4>(gs, c.base + P.o_kv, c.bars, lg, sq, c.base + P.o_state, at, t_at, t_stride, kv_base, ldf(LY(scale)));
                    else attend<1>(gs, c.base + P.o_kv, c.bars, lg, sq, c.base + P.o_state, at, t_at, t_stride, kv_base, ldf(LY(scale)));
                    kv_base += (lds32(at + 28) + kKvRows - 1) / kKvRows;
                }
                // ── merge of the shares ──
                wait_cluster(bar_of(c, kBarT), l & 1);
                if (tid == 0) mbar_expect_tx(bar_of(c, kBarT), P.n_heads * P.splits * (dh + 4) * 4);
#pragma unroll 1
                for (uint32_t kg0 = warp; kg0 < nQ; kg0 += 2 * kW) {      // two groups of 32 side by side
                    uint32_t rec[2], d[2];
                    float w[2], v[2], inv_den[2];
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        const uint32_t kg = min(kg0 + u * kW, nQ - 1), h = (kg * 32) >> P.dh_log2;
                        d[u] = (kg * 32 + lane) & (dh - 1); rec[u] = t_in + h * P.splits * (dh + 4) * 4; v[u] = 0.0f;
                        // a share's weight and maximum, one share a lane (lanes 16 .. 31 as 0 .. 15)
                        const float2 got = ldf2(rec[u] + (min(lane & 15, P.splits - 1) * (dh + 4) + dh) * 4);
                        const bool in = (lane & 15) < P.splits;
                        float m = in ? got.y : -INFINITY, gm = m;
#pragma unroll
                        for (int o = 1; o < 16; o <<= 1) gm = fmaxf(gm, __shfl_xor_sync(0xffffffffu, gm, o));
                        w[u] = m == -INFINITY ? 0.0f : expf(m - gm);
                        float den = in ? w[u] * got.x : 0.0f;
#pragma unroll
                        for (int o = 1; o < 16; o <<= 1) den += __shfl_xor_sync(0xffffffffu, den, o);
                        inv_den[u] = den > 0.0f ? 1.0f / den : 0.0f;
                    }
#pragma unroll 1
                    for (uint32_t sp = 0; sp < P.splits; sp++)
#pragma unroll
                        for (int u = 0; u < 2; u++) v[u] = fmaf(__shfl_sync(0xffffffffu, w[u], sp), ldf(rec[u] + (sp * (dh + 4) + d[u]) * 4), v[u]);
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        const uint32_t kg = kg0 + u * kW;
                        v[u] *= inv_den[u];
                        if (kg < nQ) {
                            stf(ao + (kg * 32 + lane) * 4, v[u]);
                            const float mx = warp_max(abs_or_inf(v[u]));
                            if (lane == 0) stf(ao_top + kg * 4, mx);
                            if (kg % kC == rank) {
                                ldp<float>(heads + ((kg * 32) >> P.dh_log2) * (uint32_t)sizeof(ZgClusterHead) + (uint32_t)offsetof(ZgClusterHead, attn_out))[d[u]] = v[u];
                                ldp<float>(LY(attn_buf))[kg * 32 + lane] = v[u];
                            }
                        }
                    }
                }
                workers_sync();
                x = ao; top = ao_top;
            }
            const uint32_t part = c.base + P.o_part + (ph & 1) * kW * P.seg * 128, tab = table + ph * 4 * kMaxItems;
            const uint32_t mine = stretches + (ph * kW + warp) * 8;
            matvec<FMT>(c, P, make_uint2(lds32(mine), lds32(mine + 4)), nk, c.base + P.o_lens + warp * P.list_max, x, gamma, inv, top, smax + ph * 4 * kMaxItems, part, slot, parity);
            workers_sync();
            if ((ph & 1) == 0) {
                if (ph == 0) {
                    if (lds32(c.base + kNoOperands)) return;
                    // (every warp is past the layer before)
                    if (l && warp == kW - 1 && lane == 0) mbar_arrive(bar_of(c, kBarConstEmpty + ((l - 1) & 1)));
                    // ── q | k | v to every CTA ──
#pragma unroll 1
                    for (uint32_t i = warp; i < own; i += kW) {
                        const float4 v = part_sum(part, lds32(tab + i * 4), P.seg, c4, dg);
                        const uint32_t it = lds32(items + i * 4), at = q_in + ((rank + kC * i) * 32 + c4) * 4;
#pragma unroll
                        for (uint32_t u = 0; u < 4; u++) push4(at + away[u], v, bar_of(c, kBarQ) + away[u]);
                        if (dg == 0) stg4(ldp<float>(LY(out) + (it & 255u) * 8) + (it >> 8) * 32 + c4, v);
                    }
                } else {
                    // ── activation of the CTA's pairs of columns, one column a lane ──
                    if (warp == kW - 1 && lane < kC) arrive_remote(bar_of(c, kBarGo), lane);
#pragma unroll 1
                    for (uint32_t pr = warp; 2 * pr < own; pr += kW) {
                        const float gt = pick(part_sum(part, lds32(tab + pr * 8), P.seg, c4, dg), dg), up = pick(part_sum(part, lds32(tab + pr * 8 + 4), P.seg, c4, dg), dg);
                        const uint32_t col = pr * 32 + c4 + dg, k = pair0 * 32 + col;
                        if (sec && pr != warp) ext = __ldcg(sec + pr * 32);
                        float v;
                        if (lds32(LY(act_silu))) v = __fmul_rn(gt, 1.0f / __fadd_rn(expf(-gt), ext));
                        else v = act_chain(reinterpret_cast<const ZgDecStep*>(c.smem + (LY(steps) - c.base)), lds32(LY(n_steps)), gt, up, ext, (int)lds32(LY(first_ext)), k);
                        const float hv = __fmul_rn(v, up), mx = warp_max(abs_or_inf(hv));
                        stf(hid + col * 4, hv);
                        if (lane == 0) stf(hid_top + pr * 4, mx);
                        ldp<float>(LY(out) + 32)[k] = gt; ldp<float>(LY(out) + 40)[k] = up; ldp<float>(LY(silu))[k] = v; ldp<float>(LY(hidden))[k] = hv;
                    }
                }
                if (warp < ownD && dg < 3) {      // what the norm's ops leave
                    const float4 gm = ldf4(gamma + own_i * 4);
                    const float4 b = make_float4(__fmul_rn(xown.x, inv), __fmul_rn(xown.y, inv), __fmul_rn(xown.z, inv), __fmul_rn(xown.w, inv));
                    const float4 n = make_float4(__fmul_rn(b.x, gm.x), __fmul_rn(b.y, gm.y), __fmul_rn(b.z, gm.z), __fmul_rn(b.w, gm.w));
                    static_assert(offsetof(ZgClusterLayer, grep) - offsetof(ZgClusterLayer, bare) == 16 && offsetof(ZgClusterLayer, norm) - offsetof(ZgClusterLayer, grep) == 16, "indexed by dg");
                    stg4(ldp<float>(LY(bare) + dg * 16 + ph * 4) + own_i, dg == 0 ? b : dg == 1 ? gm : n);
                }
                if (ph == 2) workers_sync();
            } else {
                // ── o | down: the owners of the residual stream's column groups ──
                const bool down = ph == 3, last = l + 1 == P.n_layers;
                const uint32_t next = c.base + P.o_const + ((l + down) & 1) * P.const_bytes;      // whose norm takes the sum
                if (down) {
                    wait_cluster(bar_of(c, kBarGo), l & 1);
                    // a column group's records are few here: its partials by the eight lanes of one dg
#pragma unroll 1
                    for (uint32_t i = warp * 4 + dg; i < own; i += 4 * kW) {
                        const uint32_t e = lds32(tab + i * 4), hi = (e >> 8) & 255u, off = mapa(c.base, i % kC) - c.base;
                        uint32_t w = e & 255u;
                        float4 v = ldf4(part + ((w * P.seg + (e >> 16)) * 32 + c4) * 4);
                        for (w++; w <= hi; w++) v = add4(v, ldf4(part + (w * P.seg * 32 + c4) * 4));
                        push4(c.base + P.o_r + ((rank * P.own_max + i / kC) * 32 + c4) * 4 + off, v, bar_of(c, kBarR) + off);
                    }
                }
                if (warp < ownD) {
                    float4 v;
                    bool next_there = true;
                    if (down) {
                        next_there = last || wait_bar(bar_of(c, kBarConstFull + ((l + 1) & 1)), ((l + 1) >> 1) & 1);
                        wait_cluster(bar_of(c, kBarR), l & 1);
                        if (tid == 0) mbar_expect_tx(bar_of(c, kBarR), ownD * 128 * min(P.F >> 5, kC));
                        const uint32_t r_in = c.base + P.o_r + ((dg * 4 * P.own_max + warp) * 32 + c4) * 4, step = P.own_max * 128;
                        v = add4(add4(ldf4(r_in), ldf4(r_in + step)), add4(ldf4(r_in + 2 * step), ldf4(r_in + 3 * step)));
                        v = shfl_add4(shfl_add4(v, 8), 16);
                    } else v = part_sum(part, lds32(tab + warp * 4), P.seg, c4, dg);
                    if (!(down && last)) {
                        // the sum, with its sum of squares and largest |x gamma|, into every CTA's inbox
                        xown = make_float4(__fadd_rn(xown.x, v.x), __fadd_rn(xown.y, v.y), __fadd_rn(xown.z, v.z), __fadd_rn(xown.w, v.w));
                        const uint32_t inbox = c.base + (down ? P.o_a1 : P.o_a2), bar = bar_of(c, down ? kBarA1 : kBarA2), grp = rank + kC * warp;
#pragma unroll
                        for (uint32_t u = 0; u < 4; u++) push4(inbox + own_i * 4 + away[u], xown, bar + away[u]);
                        const float one = pick(xown, dg), ss = warp_sum(one * one), mx = warp_max(abs_or_inf(one * ldf(next + P.blk_bytes + ((down ? 0 : P.D) + own_i + dg) * 4)));
                        if ((lane & 7) < 2) {
#pragma unroll
                            for (uint32_t u = 0; u < 4; u++) push1(inbox + (P.D + (lane & 1) * nD + grp) * 4 + away[u], lane & 1 ? mx : ss, bar + away[u]);
                        }
                        if (dg == 1 && next_there) stg4(ldp<float>(next + (uint32_t)offsetof(ZgClusterLayer, sum) + (down ? 0 : 8)) + own_i, xown);
                    }
                    if (dg == 0) stg4(ldp<float>(LY(out) + (down ? 48 : 24)) + own_i, v);
                }
            }
        }
    }
}
#undef LY

template <int FMT>
__global__ void __launch_bounds__(kThreads, 1)
k_decode_cluster(const __grid_constant__ ZgClusterPlan plan) {
    extern __shared__ __align__(128) uint8_t smem[];
    // a copy of the plan for the functions that are calls (the workers read it as constants: from shared memory a token takes 8 % longer)
    static_assert(sizeof(ZgClusterPlan) <= kDead, "the mark lies behind it");
    if (threadIdx.x < sizeof(ZgClusterPlan) / 4) reinterpret_cast<uint32_t*>(smem)[threadIdx.x] = reinterpret_cast<const uint32_t*>(&plan)[threadIdx.x];
    __syncthreads();
    const ZgClusterPlan& P = plan;
    const ZgClusterPlan* const copy = reinterpret_cast<const ZgClusterPlan*>(smem);
    Cta c;
    c.smem = smem; c.base = smem_u32(smem); c.bars = c.base + P.o_bars;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(c.rank));
    c.tid = threadIdx.x; c.lane = c.tid & 31; c.warp = c.tid >> 5;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (c.tid == 0) {
        *reinterpret_cast<uint32_t*>(smem + kDead) = *reinterpret_cast<uint32_t*>(smem + kNoOperands) = 0;
        const uint32_t nD = P.D >> 5, ownD = (nD + kC - 1 - c.rank) / kC;
#pragma unroll 1
        for (uint32_t b = kBarA1; b < kBarFull + 2 * kW * P.ring_slots; b++)
            mbar_init(bar_of(c, b), b == kBarGo ? kC : b == kBarConstEmpty || b == kBarConstEmpty + 1 ? 1 + (c.rank / P.splits < P.n_kv) : b == kBarConstFull || b == kBarConstFull + 1 ? 32 : b >= kBarKvFull && b < kBarKvEmpty ? 33 :
                                    b >= kBarKvEmpty && b < kBarFull ? 8 : 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        mbar_expect_tx(bar_of(c, kBarA1), (P.D + 2 * nD) * 4);
        mbar_expect_tx(bar_of(c, kBarQ), (P.Dq + 2 * P.Dkv) * 4);
        mbar_expect_tx(bar_of(c, kBarT), P.n_heads * P.splits * (P.dh + 4) * 4);
        mbar_expect_tx(bar_of(c, kBarA2), (P.D + 2 * nD) * 4);
        mbar_expect_tx(bar_of(c, kBarR), ownD * 128 * min(P.F >> 5, kC));
    }
    // constant parts of shared memory: planes of ones, the owners' inbox of CTAs without rows of the down weight, which warps hold an item's partials, all weights' addresses
#pragma unroll 1
    for (uint32_t i = c.tid; i < kW * 4 * 8; i += kThreads)
        *reinterpret_cast<uint32_t*>(smem + P.o_planes + (i >> 5) * kPlaneBytes + ((i >> 3) & 3) * kPlaneRow + 96 + (i & 7) * 4) = 0x01010101u;
#pragma unroll 1
    for (uint32_t i = c.tid; i < kC * P.own_max * 32; i += kThreads) reinterpret_cast<float*>(smem + P.o_r)[i] = 0.0f;
#pragma unroll 1
    for (uint32_t i = c.tid; i < P.n_layers * 7; i += kThreads)
        reinterpret_cast<unsigned long long*>(smem + P.o_ptrs)[i] = *reinterpret_cast<const unsigned long long*>(P.blocks + (size_t)(i / 7) * P.blk_bytes + (i % 7) * 8);
    Share* shares = reinterpret_cast<Share*>(smem + P.o_table);
#pragma unroll 1
    for (uint32_t i = c.tid; i < 4 * kMaxItems; i += kThreads) {
        const uint32_t ph = i / kMaxItems, it = i % kMaxItems;
        const Share s = share_of(P, c.rank, ph);
        if (it == 0) shares[ph] = s;
        uint32_t e = 0;
        if (it < s.own && s.nk) {
            const uint32_t R = s.own * s.nk, a = it * s.nk, b = a + s.nk;
            uint32_t w_lo = 0;
            while (((w_lo + 1) * R) / kW <= a) w_lo++;
            uint32_t w_hi = w_lo;
            while (((w_hi + 1) * R) / kW < b) w_hi++;
            e = w_lo | (w_hi << 8) | ((it - ((w_lo * R) / kW) / s.nk) << 16);
        }
        uint32_t* items = reinterpret_cast<uint32_t*>(shares + 4);
        items[i] = it < s.own ? item_of(P, c.rank, ph, it) : 0;
        items[4 * kMaxItems + i] = e;
    }
    // where the ranges of a scale end, a bit per record of K
    uint32_t* ranges = reinterpret_cast<uint32_t*>(smem + P.o_ranges);
#pragma unroll 1
    for (uint32_t i = c.tid; i < 4 * P.range_words; i += kThreads) ranges[i] = 0;
    __syncthreads();
    if (c.tid < 4 * kZgClusterRanges) {
        const uint32_t ph = c.tid / kZgClusterRanges, w = c.tid % kZgClusterRanges, n = (ph == 1 ? P.Dq : ph == 3 ? P.F : P.D) >> 5, S = P.splits_k[ph];
#pragma unroll 1
        for (uint32_t s = 0; s < S; s++) {
            const uint32_t end = range_end(n, S, s * kZgClusterRanges + w);
            if (end) atomicOr(ranges + ph * P.range_words + ((end - 1) >> 5), 1u << ((end - 1) & 31));
        }
    }
    __syncthreads();
    if (c.tid < kW) copy_list<FMT>(copy, c.tid);
    __syncthreads();
    cluster_sync();
    if (c.warp < kW) workers<FMT>(c, P);
    else if (c.warp == kW) weight_stream(copy);
    else {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        if (c.warp == kW + 1) {
            if (c.rank == 0 && c.lane == 0) *reinterpret_cast<volatile uint32_t*>(P.err) = 0u;
            const_stream(copy, c.rank);
        } else kv_stream(copy, c.rank);
    }
    __syncthreads();
    if (c.tid == 0 && dead()) {
        atomicExch(P.err, 1u);
        atomicAdd(&g_timeouts, 1u);
    }
    cluster_sync();      // nobody leaves while others may still store into its shared memory
    if (*reinterpret_cast<volatile uint32_t*>(P.err)) {      // a wait gave up: the step's results are not to be used, and stores to other CTAs may be under way that nobody has waited for
        __nanosleep(100000);
        cluster_sync();
        const ZgClusterLayer* ly = reinterpret_cast<const ZgClusterLayer*>(P.blocks + (size_t)(P.n_layers - 1) * P.blk_bytes);
        for (uint32_t i = c.rank * kT + c.tid; c.tid < kT && i < P.D; i += kC * kT) ly->out[6][i] = __int_as_float(0x7fc00000);
    }
}

template <int FMT>
bool launch(const ZgClusterHost& h, cudaStream_t st) {
    if (!zg_smem_limit<k_decode_cluster<FMT>>(kZgClusterSmem)) return false;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kC);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = h.plan.smem_bytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kC; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_zg_pdl ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k_decode_cluster<FMT>, h.plan);
    ZG_COUNT_LAUNCH();
    if (e != cudaSuccess) { zg_set_error("cluster decode kernel launch failed: %s", cudaGetErrorString(e)); return false; }
    return true;
}

// whether the device takes a cluster of this size (asked when a program is compiled)
template <int FMT>
bool fits(uint32_t smem) {
    if (!zg_smem_limit<k_decode_cluster<FMT>>(kZgClusterSmem)) return false;
    if (cudaFuncSetAttribute(k_decode_cluster<FMT>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) { cudaGetLastError(); return false; }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kC); cfg.blockDim = dim3(kThreads); cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kC; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k_decode_cluster<FMT>, &cfg) != cudaSuccess) { cudaGetLastError(); return false; }
    return n >= 1;
}

} // namespace

unsigned int zg_decode_cluster_timeouts() {
    unsigned int v = 0;
    cudaMemcpyFromSymbol(&v, g_timeouts, sizeof(v));
    return v;
}

// Shared memory of the plan's shape (rounded parts in order); false: a shape the kernel does not take.
bool zg_decode_cluster_layout(ZgClusterPlan& P, int fmt) {
    const uint32_t nD = P.D / 32, nQ = P.Dq / 32, nK = P.Dkv / 32, nF = P.F / 32;
    if (P.D % 32 || P.Dq % 32 || P.Dkv % 32 || P.F % 32 || (P.dh != 32 && P.dh != 64 && P.dh != 128) || P.n_layers == 0 || P.n_layers > 128) return false;
    if (P.n_kv == 0 || P.n_kv > kC || P.n_heads % P.n_kv || P.n_heads / P.n_kv > max_group(P.dh) || P.n_heads * P.dh != P.Dq || P.n_kv * P.dh != P.Dkv) return false;
    P.gs = P.n_heads / P.n_kv;
    P.dh_log2 = P.dh == 32 ? 5 : P.dh == 64 ? 6 : 7;
    P.splits = kC / P.n_kv;
    const auto up = [](uint32_t a, uint32_t b) { return (a + b - 1) / b; };
    const uint32_t pairs = up(nF, kC) + (nF % kC ? 1 : 0);      // at most, of a CTA
    const uint32_t own[4] = {up(nQ + 2 * nK, kC), up(nD, kC), 2 * pairs, nD}, nk[4] = {nD, nQ, nD, pairs};
    P.own_max = own[1];
    P.hid_max = pairs * 32;
    P.seg = 1;
    for (int ph = 0; ph < 4; ph++) {
        if (own[ph] > kMaxItems) return false;
        for (uint32_t n = 1; n <= nk[ph]; n++) {                // records of a column group may be fewer than at most
            if (ph < 3 && n != nk[ph]) continue;
            P.seg = std::max(P.seg, (up(own[ph] * n, kW) + n - 2) / n + 1);
        }
    }
    if (own[1] > kW) return false;
    uint32_t off = 256;      // the plan's own copy and the mark of a wait that gave up
    const auto put = [&](uint32_t& field, uint32_t bytes) { field = off; off += (bytes + 127) & ~127u; };
    P.const_bytes = P.blk_bytes + (2 * P.D + P.dh + 4 * kMaxItems) * 4 + 48;
    put(P.o_const, 2 * P.const_bytes);
    put(P.o_a1, (P.D + 2 * nD) * 4);
    put(P.o_a2, (P.D + 2 * nD) * 4);
    put(P.o_q, (P.Dq + 2 * P.Dkv) * 4);
    put(P.o_t, P.n_heads * P.splits * (P.dh + 4) * 4);
    put(P.o_r, kC * P.own_max * 128);
    put(P.o_part, 2 * kW * P.seg * 128);
    put(P.o_state, P.gs * kW * 4 + P.gs * kW * (P.dh + 4) * 4);
    put(P.o_sq, (P.gs + 2) * P.dh * 4);
    put(P.o_ao, (P.Dq + nQ) * 4);
    put(P.o_hid, (P.hid_max + pairs) * 4);
    put(P.o_planes, kW * kPlaneBytes);
    put(P.o_ptrs, P.n_layers * 56);
    put(P.o_table, 4 * sizeof(Share) + 8 * kMaxItems * 4 + 4 * kW * 8);
    // Copies of a warp in one layer: one for every G records and one more for each range; of n records n / (the shortest range) ranges, and two more for each column group.
    P.slot_bytes = turn_records(fmt) * record_bytes(fmt);
    P.list_max = P.range_words = 0;
    const uint32_t stride[4] = {nD, nQ, nD, nF};
    for (int ph = 0; ph < 4; ph++) {
        const uint32_t n = up(own[ph] * nk[ph], kW);
        if (stride[ph] > 255 * kZgClusterRanges || n > 0xffffu) return false;
        P.list_max += n / turn_records(fmt) + n / std::max(1u, stride[ph] / P.splits_k[ph] / kZgClusterRanges) + 2 * P.seg;
        P.range_words = std::max(P.range_words, (stride[ph] + 31) / 32);
    }
    put(P.o_ranges, 4 * P.range_words * 4);
    put(P.o_lens, kW * P.list_max);
    put(P.o_list, kW * (P.list_max * 8 + 4));
    put(P.o_bars, (kBarFull + 2 * kW * 8) * 8);
    // what is left: the keys' and values' stages, then as deep a ring as fits
    const uint32_t stage = kv_stage_bytes(P.dh);
    for (P.kv_stages = 4; P.kv_stages >= 2; P.kv_stages /= 2) {
        const uint32_t kv = P.kv_stages * stage;
        if (off + kv + 2 * kW * P.slot_bytes > kZgClusterSmem) continue;
        P.ring_slots = std::min(8u, (kZgClusterSmem - off - kv) / (kW * P.slot_bytes));
        put(P.o_kv, kv);
        put(P.o_ring, P.ring_slots * kW * P.slot_bytes);
        P.smem_bytes = off;
        switch (fmt) {
            case ZG_QFMT_I4_F16: return fits<ZG_QFMT_I4_F16>(off);
            case ZG_QFMT_I8_F16: return fits<ZG_QFMT_I8_F16>(off);
            case ZG_QFMT_I8_F32: return fits<ZG_QFMT_I8_F32>(off);
            default: return false;
        }
    }
    return false;
}

uint32_t zg_decode_cluster_turns(const ZgClusterPlan& P, int fmt) {
    const uint32_t n[4] = {P.D / 32, P.Dq / 32, P.D / 32, P.F / 32}, G = turn_records(fmt);
    uint32_t most = 0;
    for (uint32_t r = 0; r < kC; r++) {
        uint32_t turns = 0;
        for (uint32_t ph = 0; ph < 4; ph++) {
            const Share s = share_of(P, r, ph);
            uint32_t at = 0, of_group = 0;      // ranges' ends, and the turns of what lies in this CTA's part of a column group
            for (uint32_t i = 1; i <= P.splits_k[ph] * kZgClusterRanges; i++) {
                const uint32_t end = range_end(n[ph], P.splits_k[ph], i - 1), lo = std::max(at, s.k0), hi = std::min(end, s.k0 + s.nk);
                if (hi > lo) of_group += (hi - lo + G - 1) / G;
                at = end;
            }
            turns += s.own * of_group;
        }
        most = std::max(most, turns);
    }
    return most;
}

// Which weight (0 .. 6) and column group the items of the CTAs are, [rank][phase][kZgClusterItems], -1: none.
void zg_decode_cluster_items(const ZgClusterPlan& P, int* weight, uint32_t* group) {
    for (uint32_t r = 0; r < kC; r++)
        for (uint32_t ph = 0; ph < 4; ph++) {
            const Share s = share_of(P, r, ph);
            for (uint32_t i = 0; i < kMaxItems; i++) {
                const uint32_t at = (r * 4 + ph) * kMaxItems + i, it = i < s.own ? item_of(P, r, ph, i) : 0;
                weight[at] = i < s.own ? (int)(it & 255u) : -1;
                group[at] = it >> 8;
            }
        }
}

bool zg_decode_cluster_launch(const ZgClusterHost& h, cudaStream_t st) {
    switch (h.fmt) {
        case ZG_QFMT_I4_F16: return launch<ZG_QFMT_I4_F16>(h, st);
        case ZG_QFMT_I8_F16: return launch<ZG_QFMT_I8_F16>(h, st);
        default: return launch<ZG_QFMT_I8_F32>(h, st);
    }
}

void zg_decode_cluster_free(ZgClusterHost* h) {
    cudaFree(h->d_blocks); cudaFree(h->d_smax); cudaFree(h->d_err);
    if (h->h_err) cudaFreeHost(h->h_err);
    *h = ZgClusterHost();
}
