// Attention of many query rows over f32 keys and values on the 5th-generation tensor cores, with f32 accuracy.
//
// Every f32 operand x is split into two half-precision values, x = hi + lo: hi = f16(x s), lo = f16(x s - hi), with s a power of
// two that brings the largest magnitude of its tile (keys, values) or row (queries) to [2^14, 2^15).  hi and lo together keep 22
// to 24 significant bits of everything within 2^-17 of that maximum (what is smaller loses bits below 2^-39 of the maximum), so
// the split costs about one f32 rounding per operand.  A product is three MMAs, hi lo + lo hi + hi hi, accumulated in f32 in TMEM: the
// small cross terms first, so that only the dk / 16 steps of hi hi add to a large accumulator.  The probabilities (at most 1) are
// scaled by 2^14 and split the same way.  Outputs of different key tiles are added in registers, in f32.
//
//   * k_atc_prep: 128 keys (or 128 columns of 128 values) per CTA, held in registers: maximum, split, store.  Keys as rows [hi dims | lo
//     dims], values transposed, rows of one value column over all keys [hi | lo]: both are K-major operands that TMA brings as they lie (128-byte
//     swizzle).  The cache is read and split once per step instead of once per query tile that meets it.
//   * k_attention_tc: one CTA per 128 query rows.  Warp 16 loads 16 KB pieces through a ring of 12, warp 17 issues
//     tcgen05.mma.cta_group::1.kind::f16, warps 0 - 15 are the softmax: four threads share a query row, each with a quarter of the tile's keys
//     and a quarter of the output columns.  Queries lie split in TMEM (A operand), scores of two key tiles alternate between two TMEM buffers, and
//     the probabilities replace the scores they came from, in place, as the A operand of the product with the values: no operand but keys and values
//     passes through shared memory, whose bandwidth (128 B per clock) a 128 x 128 tile with both operands in it would saturate.  MMA order:
//     scores of tile i + 1 before values of tile i, so the softmax of one tile runs beside the products of its neighbours.
//   * Measured per 128 x 128 tile of 128 dims (its 48 MMAs execute in 3072 clocks): 9400 clocks with one thread per query row and the MMAs issued
//     inside a single lane's branch, 9100 with four threads per row, 4700 once the whole MMA warp walks the tiles (below).
//   * Every wait is bounded; a CTA whose wait ran out counts it (zg_attention_tc_timeouts), stops issuing, makes NaN of its rows and frees its TMEM.
//
// What pairs cannot hold is evaluated in plain f32 (atc_plain: the CTA's 512 softmax threads over f32 tiles, as the SIMT kernels do it; 1.3 times
// their time): all rows of an op with more keys than there are planes for, and of a CTA that met a key or value tile, or a query row, that holds
// something non-finite or whose magnitudes lie too far apart for one scale (is_small; such a tile is marked by a NaN scale), whose scores all lie
// near the lowest float (a mask of such values), or whose scaled products or outputs could leave f32's range before the scales are undone (queries
// times keys beyond 2^108, values beyond 2^94).
#include "attention_tc.cuh"
#include "split_tc.cuh"

#include <algorithm>
#include <map>
#include <type_traits>
#include <vector>

namespace {

constexpr uint32_t kAtcThreads = 576, kAtcRing = 12, kAtcPiece = 16384;
constexpr uint32_t kAtcShare = 2 * 4 * 128 * 4;                   // row maxima of the four quarters, two tiles
constexpr uint32_t kAtcTiles = 512;                               // key tiles whose class and scales a CTA keeps at hand
constexpr uint32_t kAtcSmem = kAtcRing * kAtcPiece + kAtcShare + kAtcTiles * 12 + 1024 + 256;
constexpr float kNotANumber = __builtin_nanf("");
constexpr size_t kAtcProgramKeys = 1u << 20;                      // the most keys that a DeviceOp.attention batch lays out planes for
constexpr float kFltMax = 3.4028234e38f, kAtcLow = -1e36f;          // a row whose largest score is below kAtcLow is evaluated in plain f32
constexpr float kAtcBig = 1.2e24f;                                // 2^80: scores are at most 2^38 times f, outputs 2^33 times v_inv, and stay finite below it
constexpr float kLog2e = 1.4426950408889634f, kLn2 = 0.6931471805599453f;
constexpr float kPScale = 16384.0f, kPInv = 1.0f / 16384.0f;      // probabilities are held times 2^14

__device__ __forceinline__ float ex2(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
// A scaled element that is not zero but below 2^-18 of the largest magnitude its scale is made for (which is brought to [2^14, 2^15)).  A pair keeps it to
// 2^-40 of that magnitude, fewer than 22 bits of its own: where that many are small, it is their own size that counts (values of a column that is small
// as a whole, a key beside one that no row sees), not what they add to the large ones.  Normally distributed tiles of 128 x 128 have 0.1 to 0.3 of them.
constexpr uint32_t kAtcSmallTile = 24, kAtcSmallQuery = 3;          // of 128 keys or values, of a quarter row
__device__ __forceinline__ uint32_t is_small(float x, float scale) { const float a = fabsf(x * scale); return a < 0.0625f && a > 0.0f ? 1u : 0u; }
// a score in units of log2 and what is added to it in natural units.  A finite term does not mask: near the lowest float, where times log2(e) it would be
// -inf, the result stays finite, and a row without any higher score is evaluated in plain f32.
__device__ __forceinline__ float plus_natural(float x, float v) {
    const float y = fmaf(v, kLog2e, x);
    return y < -kFltMax && v >= -kFltMax ? -kFltMax : y;
}
// ── where keys, values and queries come from ─────────────────────────────────────────────────────────────────────
// A SOURCE names the keys of a step (for k_atc_prep) and, for the attention kernel, a CTA's items and range of key tiles, the class of a tile
// (0: no row sees it, 1: every row sees all of it, 2: some), a row's query and what becomes of its scores.  Keys are counted from the first one
// that any row of the step can see.

// CACHED_ATTENTION: rows are (token, head of the key group) pairs
template <bool EXTRA>      // score caps, score tables, sigmoid weights, pooled blocks
struct AtcCached {
    CaArgs a;
    uint32_t rh, row_tiles, n_vs, vslice, splits, tiles;      // tiles: of 128 keys, that the planes have room for
    float* part;
    struct Step { uint32_t pos0, slot, k_lo, n_pool, n_keys; };
    __device__ __forceinline__ Step step() const {
        Step s;
        s.pos0 = (uint32_t)ctl_word(a.ctl, ZG_CTL_POS); s.slot = ca_slot(a);
        s.k_lo = mask_low(s.pos0, a.kind, a.size);
        const uint32_t last = s.pos0 + a.T - 1;
        s.n_pool = EXTRA && a.pool ? min(pooled_seen(last, a.size, a.pool), a.pool_rows) : 0u;
        s.n_keys = min(s.n_pool + last - s.k_lo + 1, tiles * 128);
        return s;
    }
    // row `u` of a key item or a value head; u < n_keys
    __device__ __forceinline__ const float* row(const Step& s, bool value, uint32_t item, uint32_t u) const {
        const uint32_t col = item * (value ? a.dv : a.dk), w = value ? a.vw : a.kw;
        if (EXTRA && u < s.n_pool) return (value ? a.vp : a.kp) + (size_t)s.slot * a.pool_rows * a.kw + (size_t)u * a.kw + col;
        return (value ? a.vc + a.v_off : a.kc + a.k_off) + ((size_t)s.slot * a.R + (s.k_lo + u - s.n_pool) % a.R) * w + col;
    }
    __device__ __forceinline__ uint32_t prep_keys(uint32_t) const { return step().n_keys; }
    struct Cta { Step s; uint32_t r0, nq, p_min, p_max, lo_min, lo_max, nb_min, nb_max, gm, g, m, vs, split, used, t0, t1; };
    __device__ __forceinline__ Cta cta(uint32_t bk) const {
        Cta c;
        c.s = step();
        const uint32_t items = a.G * a.maps * n_vs, item = blockIdx.x % items;
        c.gm = item / n_vs; c.vs = item % n_vs; c.g = c.gm / a.maps; c.m = c.gm % a.maps; c.split = blockIdx.y;
        c.r0 = (row_tiles - 1 - blockIdx.x / items) * 128;            // later rows meet more keys: heaviest first
        c.nq = min(128u, a.T * rh - c.r0);
        c.p_min = c.s.pos0 + c.r0 / rh; c.p_max = c.s.pos0 + (c.r0 + c.nq - 1) / rh;
        c.lo_min = mask_low(c.p_min, a.kind, a.size); c.lo_max = mask_low(c.p_max, a.kind, a.size);
        c.nb_min = c.nb_max = 0;
        if (EXTRA && a.pool) { c.nb_min = pooled_seen(c.p_min, a.size, a.pool); c.nb_max = pooled_seen(c.p_max, a.size, a.pool); }
        const uint32_t first = c.s.n_pool ? 0u : (c.lo_min - c.s.k_lo) / bk, end = (min(c.s.n_keys, c.s.n_pool + c.p_max - c.s.k_lo + 1) + bk - 1) / bk;
        // at most a share per key tile, whatever the capacity asks for: the merge reads a record per share
        const uint32_t n = end - min(end, first);
        c.used = max(1u, min(splits, n));
        const uint32_t per = (n + c.used - 1) / c.used;
        c.t0 = min(end, first + c.split * per); c.t1 = min(end, c.t0 + per);
        return c;
    }
    __device__ __forceinline__ uint32_t plain_end(const Cta& c, uint32_t bk) const { return c.t1 * bk; }
    __device__ __forceinline__ bool idle(const Cta& c) const { return c.split >= c.used; }       // a share that the step has no keys for
    __device__ __forceinline__ bool over(const Cta&) const { return false; }
    __device__ __forceinline__ uint32_t k_item(const Cta& c) const { return c.gm; }
    __device__ __forceinline__ uint32_t v_item(const Cta& c) const { return c.g * n_vs + c.vs; }
    __device__ __forceinline__ uint32_t classify(const Cta& c, uint32_t t, uint32_t bk) const {
        const uint32_t u0 = t * bk, u1 = u0 + bk - 1;
        if (EXTRA && u0 < c.s.n_pool) {
            if (u1 >= c.s.n_pool) return 2;
            return u0 >= c.nb_max ? 0 : u1 < c.nb_min ? 1 : 2;
        }
        const uint32_t j0 = c.s.k_lo + u0 - c.s.n_pool, j1 = j0 + bk - 1;
        if (j0 > c.p_max || j1 < c.lo_min) return 0;
        return j1 <= c.p_min && j0 >= c.lo_max && u1 < c.s.n_keys ? 1 : 2;
    }
    struct Row { bool on; uint32_t r, p, lo, nb, hm; const float* tab; };
    __device__ __forceinline__ Row query(const Cta& c, uint32_t i) const {
        Row w;
        w.on = i < c.nq;
        w.r = c.r0 + (w.on ? i : 0);
        const uint32_t t = w.r / rh, h = c.g * rh + w.r % rh;
        w.hm = h * a.maps + c.m;
        w.p = c.s.pos0 + t; w.lo = mask_low(w.p, a.kind, a.size);
        w.nb = EXTRA && a.pool ? pooled_seen(w.p, a.size, a.pool) : 0u;
        w.tab = EXTRA && a.tab ? a.tab + (size_t)w.hm * a.tab_rs : nullptr;
        return w;
    }
    __device__ __forceinline__ const float* q_row(const Cta& c, const Row& w) const { return a.q + (size_t)(w.r / rh) * a.q_rs + a.q_off + (size_t)w.hm * a.dk; }
    __device__ __forceinline__ uint32_t dk() const { return a.dk; }
    __device__ __forceinline__ uint32_t dv(const Cta& c) const { return min(vslice, a.dv - c.vs * vslice); }
    __device__ __forceinline__ float scale(const Cta&) const { return a.scale; }
    __device__ __forceinline__ bool sigmoid() const { return EXTRA && a.wkind; }
    __device__ __forceinline__ bool plain_tile() const { return !EXTRA; }
    // scores in units of log2 of keys u0 .. u0 + N - 1, from the scaled products times log2(e); -inf where the row does not see the key
    template <int N>
    __device__ __forceinline__ void scores(const Cta& c, const Row& w, uint32_t, uint32_t u0, uint32_t, float (&x)[N]) const {
        if (EXTRA && a.cap > 0.0f) {
#pragma unroll
            for (int i = 0; i < N; i++) x[i] = a.cap * tanhf(x[i] * kLn2 / a.cap) * kLog2e;
        }
        if (EXTRA && w.tab) {                                         // no pooled blocks here: positions ascend with u
            const uint32_t j0 = c.s.k_lo + u0;
#pragma unroll
            for (int i = 0; i < N; i++) if (j0 + i <= w.p && j0 + i >= w.lo) x[i] = plus_natural(x[i], w.tab[w.p - j0 - i]);
        }
        const uint32_t base = c.s.k_lo - c.s.n_pool;
#pragma unroll
        for (int i = 0; i < N; i++) {
            const uint32_t u = u0 + i, j = base + u;
            const bool seen = EXTRA && u < c.s.n_pool ? u < w.nb : u < c.s.n_keys && j <= w.p && j >= w.lo;
            if (!seen) x[i] = -INFINITY;
        }
    }
    // natural units, from the plain product
    __device__ __forceinline__ float slow_score(const Cta& c, const Row& w, uint32_t u, float dot) const {
        const bool pooled = EXTRA && u < c.s.n_pool;
        const uint32_t j = c.s.k_lo + u - c.s.n_pool;
        if (pooled ? u >= w.nb : (u >= c.s.n_keys || j > w.p || j < w.lo)) return -INFINITY;
        float s = ca_score(a, dot);
        if (EXTRA && w.tab && !pooled) s += w.tab[w.p - j];
        return s;
    }
    // What a row's outputs are multiplied by; sums and outputs carry the factor 1 / unit, `m` is in natural or (m2) log2 units.  A share of the keys
    // leaves its maximum and sum for the merge (`first`: one of the row's threads).
    __device__ __forceinline__ float finish(const Cta& c, const Row& w, bool first, float m, bool m2, float l, float unit) const {
        if (splits > 1) {
            if (first && c.vs == 0) {
                float* mine = part + (((size_t)(w.r / rh) * a.H * a.maps + w.hm) * splits + c.split) * (4 + a.dv);
                mine[0] = sigmoid() ? 0.0f : m2 ? m * kLn2 : m; mine[1] = l * unit;
            }
            return unit;
        }
        if (sigmoid()) return unit * a.out_scale;
        float sum = l * unit;
        if (a.sink) sum += m2 ? exp2f(fmaf(ca_sink(a, w.hm), kLog2e, -m)) : expf(ca_sink(a, w.hm) - m);
        return unit * a.out_scale / sum;
    }
    // the record of a share without keys weighs nothing
    __device__ __forceinline__ void leave_empty(const Cta& c, uint32_t i) const {
        const Row w = query(c, i);
        if (!w.on || c.vs) return;
        float* mine = part + (((size_t)(w.r / rh) * a.H * a.maps + w.hm) * splits + c.split) * (4 + a.dv);
        mine[0] = -INFINITY; mine[1] = 0.0f;
    }
    // four finished output columns from col on
    __device__ __forceinline__ void put(const Cta& c, const Row& w, uint32_t col, float4 v) const {
        if (col >= dv(c)) return;                                     // a multiple of four, as col is
        const size_t t = w.r / rh, at = (size_t)c.vs * vslice + col;
        float* out = splits == 1 ? a.dst + t * a.dst_rs + (size_t)w.hm * a.dv + at : part + ((t * a.H * a.maps + w.hm) * splits + c.split) * (4 + a.dv) + 4 + at;
        if ((reinterpret_cast<uintptr_t>(out) & 15) == 0) *reinterpret_cast<float4*>(out) = v;
        else { out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w; }
    }
};

// DeviceOp.attention of a prompt (reference src/backend/reference.zig:599-671): one table entry per head, an additive mask in memory.  Entries
// that read the same keys and values share their planes, entries with the same mask its tile classes.
struct AtcProgram {
    const ZgBatchEntry* tab;
    const uint32_t* dyn;
    const uint32_t* map;        // [count] planes of an entry, [count] its mask, [kv items] and [mask items] an entry that stands for the item
    uint32_t count, kv_items, mask_items, seq_q, head, row_tiles, tiles;
    uint8_t* classes;           // [mask items][row tiles][tiles]: what k_atc_masks found
    uint32_t* bits;             // [mask items][row tiles][tiles][128 rows][4]: which keys of a tile a row sees
    __device__ __forceinline__ const ZgBatchEntry& kv_entry(uint32_t item) const { return tab[map[2 * count + item]]; }
    // keys that any entry of the item (offset 0: planes, `count`: masks) attends over; whole warps call it together
    __device__ __forceinline__ uint32_t item_keys(uint32_t item, uint32_t offset) const {
        uint32_t n = 0;
        for (uint32_t i = threadIdx.x & 31; i < count; i += 32) if (map[offset + i] == item) n = max(n, dyn[tab[i].dyn]);
        return min(__reduce_max_sync(0xffffffffu, n), tiles * 128);
    }
    __device__ __forceinline__ uint32_t prep_keys(uint32_t item) const { return item_keys(item, 0); }
    struct Cta { const ZgBatchEntry* e; const uint8_t* cls; const uint32_t* bits; uint32_t r0, nq, n_keys, n_all, kv, t0, t1; bool masked; };
    __device__ __forceinline__ Cta cta(uint32_t bk) const {
        Cta c;
        const uint32_t item = blockIdx.x % count, tile = row_tiles - 1 - blockIdx.x / count;      // under a causal mask later rows meet more keys
        c.e = tab + item;
        c.kv = map[item];
        c.masked = c.e->u[0] != 0;
        const size_t m = ((size_t)map[count + item] * row_tiles + tile) * tiles;
        c.cls = classes + m; c.bits = bits + m * 512;
        c.r0 = tile * 128; c.nq = min(128u, seq_q - c.r0);
        c.n_keys = min(dyn[c.e->dyn], tiles * 128);
        c.n_all = dyn[c.e->dyn];
        c.t0 = 0; c.t1 = (c.n_keys + bk - 1) / bk;
        return c;
    }
    __device__ __forceinline__ uint32_t plain_end(const Cta& c, uint32_t) const { return c.n_all; }
    __device__ __forceinline__ bool idle(const Cta&) const { return false; }
    __device__ __forceinline__ void leave_empty(const Cta&, uint32_t) const {}
    __device__ __forceinline__ bool over(const Cta& c) const { return c.n_all > c.n_keys; }          // more keys than there are planes for
    __device__ __forceinline__ uint32_t k_item(const Cta& c) const { return c.kv; }
    __device__ __forceinline__ uint32_t v_item(const Cta& c) const { return c.kv; }
    __device__ __forceinline__ uint32_t classify(const Cta& c, uint32_t t, uint32_t bk) const {
        const uint32_t k = c.masked ? c.cls[t * bk / 128] : 1u;
        return k == 1 && (t + 1) * bk > c.n_keys ? 2u : k;
    }
    struct Row { bool on; uint32_t r; };
    __device__ __forceinline__ Row query(const Cta& c, uint32_t i) const {
        Row w;
        w.on = i < c.nq;
        w.r = c.r0 + (w.on ? i : 0);
        return w;
    }
    __device__ __forceinline__ const float* q_row(const Cta& c, const Row& w) const { return c.e->s0 + c.e->u[3] + (size_t)w.r * c.e->u[9]; }
    __device__ __forceinline__ const float* mask_row(const Cta& c, const Row& w) const { return c.masked ? c.e->s3 + c.e->u[6] + (size_t)w.r * c.e->u[15] : nullptr; }
    __device__ __forceinline__ uint32_t dk() const { return head; }
    __device__ __forceinline__ uint32_t dv(const Cta&) const { return head; }
    __device__ __forceinline__ float scale(const Cta& c) const { return c.e->f; }
    __device__ __forceinline__ bool sigmoid() const { return false; }
    __device__ __forceinline__ bool plain_tile() const { return true; }
    // tile 2: keys seen or not, as the bits say; tile 3: the mask's values are added, four at a time (all at once they would not fit the registers)
    template <int N>
    __device__ __forceinline__ void scores(const Cta& c, const Row& w, uint32_t t, uint32_t u0, uint32_t cls, float (&x)[N]) const {
        uint32_t seen = 0xffffffffu;                                  // of the 32 keys that hold u0 .. u0 + N - 1
        if (c.masked) seen = c.bits[(size_t)(u0 >> 7) * 512 + (w.r - c.r0) * 4 + ((u0 >> 5) & 3)] >> (u0 & 31);
#pragma unroll
        for (int i = 0; i < N; i++) if (!((seen >> i) & 1) || u0 + i >= c.n_keys) x[i] = -INFINITY;
        if (cls < 3) return;
        const float* mask = mask_row(c, w) + (size_t)u0 * c.e->u[14];
        const uint32_t rs = c.e->u[14];
#pragma unroll
        for (int i = 0; i < N; i += 4) {
            float v[4];
#pragma unroll
            for (int j = 0; j < 4; j++) { v[j] = u0 + i + j < c.n_keys ? *mask : 0.0f; mask += rs; }
#pragma unroll
            for (int j = 0; j < 4; j++) x[i + j] = x[i + j] == -INFINITY ? -INFINITY : plus_natural(x[i + j], v[j]);
            asm volatile("" ::: "memory");
        }
    }
    __device__ __forceinline__ float slow_score(const Cta& c, const Row& w, uint32_t u, float dot) const {
        if (u >= c.n_all) return -INFINITY;
        float s = dot * c.e->f;
        if (c.masked) {
            const float mv = mask_row(c, w)[(size_t)u * c.e->u[14]];
            if (!isfinite(mv)) return -INFINITY;
            s += mv;
        }
        return isfinite(s) ? s : -INFINITY;      // a non-finite score counts as masked, as in the reference
    }
    __device__ __forceinline__ float finish(const Cta&, const Row&, bool, float, bool, float l, float) const { return l > 0.0f ? 1.0f / l : 0.0f; }
    __device__ __forceinline__ void put(const Cta& c, const Row& w, uint32_t col, float4 v) const {
        float* out = c.e->dst + c.e->u[7] + (size_t)w.r * c.e->u[17] + col;
        if ((reinterpret_cast<uintptr_t>(out) & 15) == 0) *reinterpret_cast<float4*>(out) = v;
        else { out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w; }
        if (!c.e->dst2) return;
        const size_t rs = c.e->d2_rs;
        out = c.e->dst2 + c.e->d2_off + (size_t)w.r * c.e->d2_cs + col * rs;
        if (rs == 1 && (reinterpret_cast<uintptr_t>(out) & 15) == 0) *reinterpret_cast<float4*>(out) = v;
        else { out[0] = v.x; out[rs] = v.y; out[2 * rs] = v.z; out[3 * rs] = v.w; }
    }
};
template <bool EXTRA>
__device__ __forceinline__ const float* src_row(const AtcCached<EXTRA>& s, bool value, uint32_t head, uint32_t u) { return s.row(s.step(), value, head, u); }
template <bool EXTRA>
__device__ __forceinline__ const float* src_key(const AtcCached<EXTRA>& s, const typename AtcCached<EXTRA>::Cta& c, uint32_t u) { return s.row(c.s, false, c.gm, u); }
template <bool EXTRA>
__device__ __forceinline__ const float* src_value(const AtcCached<EXTRA>& s, const typename AtcCached<EXTRA>::Cta& c, uint32_t u) { return s.row(c.s, true, c.g, u) + c.vs * s.vslice; }

__device__ __forceinline__ const float* src_row(const AtcProgram& s, bool value, uint32_t item, uint32_t u) {
    const ZgBatchEntry& e = s.kv_entry(item);
    return value ? e.s2 + e.u[5] + (size_t)u * e.u[13] : e.s1 + e.u[4] + (size_t)u * e.u[11];
}
__device__ __forceinline__ const float* src_key(const AtcProgram&, const AtcProgram::Cta& c, uint32_t u) { return c.e->s1 + c.e->u[4] + (size_t)u * c.e->u[11]; }
__device__ __forceinline__ const float* src_value(const AtcProgram&, const AtcProgram::Cta& c, uint32_t u) { return c.e->s2 + c.e->u[5] + (size_t)u * c.e->u[13]; }

struct AtcPlanes {
    __half* k;           // [key items][tiles * 128][2 dkp]: hi | lo of a key
    __half* v;           // [value items][vslice][2 tiles * 128]: hi | lo of a value column; an item is a slice of a value head's columns
    float* k_inv;        // [key items][tiles]: 1 / scale of a tile, NaN where it holds something non-finite
    float* v_inv;
    uint32_t dkp, vslice, dk, dv, k_items, v_items, n_vs, tiles;
};

// CTA (x, item): 128 keys of key item y at a time, or 128 values of value item y - k_items.  C: 64-wide chunks of the widest item, all of which lie in
// registers: every load is in flight at once.  (Reading twice, once for the maximum, took 17.5 us where this takes 9.5: 2048 keys and values of
// 4 heads of 128, cold.)
constexpr uint32_t kPrepThreads = 512;
template <class Src, int C>
__global__ void __launch_bounds__(kPrepThreads, C == 1 ? 3 : C == 2 ? 2 : 1) k_atc_prep(const Src src, const AtcPlanes pl) {
    pdl_enter();
    __shared__ float red[kPrepThreads / 32];
    __shared__ uint32_t n_small[kPrepThreads / 32];
    __shared__ uint32_t t_hi[64][65], t_lo[64][65];      // a 64-column chunk of 128 values, transposed: pairs of keys per word
    const bool value = blockIdx.y >= pl.k_items;
    const uint32_t item = value ? blockIdx.y - pl.k_items : blockIdx.y, head = value ? item / pl.n_vs : item, n_keys = src.prep_keys(head);
    const uint32_t first = value ? item % pl.n_vs * pl.vslice : 0, dim = value ? min(pl.vslice, pl.dv - first) : pl.dk, padded = value ? pl.vslice : pl.dkp;
    const uint32_t tid = threadIdx.x, c4 = 4 * (tid & 15), k0 = 4 * (tid >> 4);      // columns c4 .. + 3 of every chunk, keys k0 .. + 3
    // CTAs for four per SM; they take the tiles that hold keys in turn (a step's capacity may be many times its length)
#pragma unroll 1
    for (uint32_t tile = blockIdx.x; tile * 128 < n_keys; tile += gridDim.x) {
        const uint32_t u0 = tile * 128;
        if (tile != blockIdx.x) __syncthreads();         // the tile before is done with the shared memory
        float4 x[C][4];
        float mx = 0.0f;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t u = u0 + k0 + k;
            const float* row = u < n_keys ? src_row(src, value, head, u) + first : nullptr;
#pragma unroll
            for (int c = 0; c < C; c++) x[c][k] = row && 64 * c + c4 < dim ? *reinterpret_cast<const float4*>(row + 64 * c + c4) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
#pragma unroll
        for (int c = 0; c < C; c++)
#pragma unroll
            for (int k = 0; k < 4; k++) mx = abs_or_inf(abs_or_inf(abs_or_inf(abs_or_inf(mx, x[c][k].x), x[c][k].y), x[c][k].z), x[c][k].w);
        mx = warp_max(mx);
        if ((tid & 31) == 0) red[tid >> 5] = mx;
        __syncthreads();
        mx = warp_max(red[tid & 15]);
        float scale, inv;
        split_scale(mx, scale, inv);
        uint32_t small = 0;
#pragma unroll
        for (int c = 0; c < C; c++)
#pragma unroll
            for (int k = 0; k < 4; k++) small += is_small(x[c][k].x, scale) + is_small(x[c][k].y, scale) + is_small(x[c][k].z, scale) + is_small(x[c][k].w, scale);
        small = __reduce_add_sync(0xffffffffu, small);
        if ((tid & 31) == 0) n_small[tid >> 5] = small;
        __syncthreads();
        if (tid == 0) {
            small = 0;
            for (uint32_t i = 0; i < kPrepThreads / 32; i++) small += n_small[i];
            if (small >= min(kAtcSmallTile, max(4u, min(128u, n_keys - u0)))) inv = __uint_as_float(0x7fffffffu);
            (value ? pl.v_inv : pl.k_inv)[(size_t)item * pl.tiles + tile] = inv;
        }
#pragma unroll
        for (int c = 0; c < C; c++) {
            if (64 * c >= padded) break;
            if (!value) {
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    uint32_t h[2], l[2];
                    split2(x[c][k].x * scale, x[c][k].y * scale, h[0], l[0]);
                    split2(x[c][k].z * scale, x[c][k].w * scale, h[1], l[1]);
                    __half* out = pl.k + ((size_t)item * pl.tiles * 128 + u0 + k0 + k) * 2 * pl.dkp + 64 * c + c4;
                    *reinterpret_cast<uint2*>(out) = make_uint2(h[0], h[1]);
                    *reinterpret_cast<uint2*>(out + pl.dkp) = make_uint2(l[0], l[1]);
                }
                continue;
            }
            if (c) __syncthreads();
#pragma unroll
            for (int k = 0; k < 4; k += 2) {
                const float* a = &x[c][k].x;
                const float* b = &x[c][k + 1].x;
#pragma unroll
                for (int e = 0; e < 4; e++) split2(a[e] * scale, b[e] * scale, t_hi[c4 + e][(k0 + k) / 2], t_lo[c4 + e][(k0 + k) / 2]);
            }
            __syncthreads();
#pragma unroll
            for (uint32_t i = tid; i < 64 * 64; i += kPrepThreads) {
                const uint32_t col = i >> 6, w = i & 63;
                uint32_t* out = reinterpret_cast<uint32_t*>(pl.v + ((size_t)item * pl.vslice + 64 * c + col) * 2 * pl.tiles * 128 + u0);
                out[w] = t_hi[col][w];
                out[pl.tiles * 64 + w] = t_lo[col][w];
            }
        }
    }
}

// A mask's 128 x 128 tiles: which entries are finite (bits), and the tile's class: 0 none, 1 all, and zero, 2 those that are are zero, 3 anything
// else.  CTA (key tile, row tile, mask item); a warp takes eight rows, lane l of it keys l, l + 32, l + 64, l + 96, all loads in flight at once.
__global__ void __launch_bounds__(512) k_atc_masks(const AtcProgram src) {
    pdl_enter();
    const ZgBatchEntry& e = src.tab[src.map[2 * src.count + src.kv_items + blockIdx.z]];
    const uint32_t u0 = blockIdx.x * 128, r0 = blockIdx.y * 128, n_keys = src.item_keys(blockIdx.z, src.count), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (u0 >= n_keys) return;
    const float* mask = e.s3 + e.u[6];
    const size_t tile = ((size_t)blockIdx.z * src.row_tiles + blockIdx.y) * src.tiles + blockIdx.x;
    float v[8][4];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t u = u0 + 32 * k + lane, r = r0 + 8 * warp + i;
            v[i][k] = u < n_keys && r < src.seq_q ? mask[(size_t)u * e.u[14] + (size_t)r * e.u[15]] : 0.0f;      // what lies outside changes no class
        }
    bool any = false, all = true, zero = true;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        uint32_t word = 0;
        const bool row = r0 + 8 * warp + i < src.seq_q;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const bool fin = isfinite(v[i][k]);
            const uint32_t b = __ballot_sync(0xffffffffu, fin);
            if (lane == k) word = b;
            any = any || (fin && row && u0 + 32 * k + lane < n_keys);
            all = all && fin;
            zero = zero && (!fin || v[i][k] == 0.0f);
        }
        if (lane < 4) src.bits[tile * 512 + (8 * warp + i) * 4 + lane] = word;
    }
    const int a = __syncthreads_or(any), f = __syncthreads_and(all), z = __syncthreads_and(zero);
    if (threadIdx.x == 0) src.classes[tile] = !a ? 0 : !z ? 3 : f ? 1 : 2;
}

// The CTA's rows in plain f32, by its 512 softmax threads once the ring is idle: thread (ty, tx) of 32 x 16 holds rows 4 ty .. + 3 against keys tx + 16 c of 64, and value
// columns tx + 16 c.  Keys that a row does not see are left out of its sums (what they hold need not be finite).
template <int DV, class Src>
__device__ __noinline__ void atc_plain(const Src& src, const typename Src::Cta& c, uint32_t bk, float* sm) {
    constexpr int OC = DV / 16, KP = 68;
    float* const Qs = sm;                              // [128][64]: 64 dims of the queries, of the keys
    float* const Ks = Qs + 128 * 64;                   // [64][68]
    float* const Ps = Ks + 64 * KP;                    // [128][68]: probabilities
    float* const Vs = Ps + 128 * KP;                   // [64][DV]
    const uint32_t tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, dk = src.dk(), dv = src.dv(c);
    float o[4][OC], m[4], l[4];
#pragma unroll
    for (int r = 0; r < 4; r++) {
        m[r] = -INFINITY; l[r] = 0.0f;
#pragma unroll
        for (int k = 0; k < OC; k++) o[r][k] = 0.0f;
    }
#pragma unroll 1
    for (uint32_t u0 = c.t0 * bk; u0 < src.plain_end(c, bk); u0 += 64) {
        if (u0 / bk < c.t1 && !src.classify(c, u0 / bk, bk)) continue;
        float sc[4][4];
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int k = 0; k < 4; k++) sc[r][k] = 0.0f;
#pragma unroll 1
        for (uint32_t d0 = 0; d0 < dk; d0 += 64) {
            bar_sync(5, 512);                          // the readers of the slice, the probabilities and the values before are done
            for (uint32_t i = tid; i < 128 * 16; i += 512) {
                const uint32_t r = i >> 4, d = 4 * (i & 15);
                *reinterpret_cast<float4*>(Qs + r * 64 + d) = r < c.nq && d0 + d < dk ? *reinterpret_cast<const float4*>(src.q_row(c, src.query(c, r)) + d0 + d) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
            for (uint32_t i = tid; i < 64 * 16; i += 512) {
                const uint32_t r = i >> 4, d = 4 * (i & 15);
                *reinterpret_cast<float4*>(Ks + r * KP + d) = u0 + r < src.plain_end(c, bk) && d0 + d < dk ? *reinterpret_cast<const float4*>(src_key(src, c, u0 + r) + d0 + d) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
            if (d0 == 0)
                for (uint32_t i = tid; i < 64 * (DV / 4); i += 512) {
                    const uint32_t r = i / (DV / 4), col = 4 * (i % (DV / 4));
                    *reinterpret_cast<float4*>(Vs + r * DV + col) = u0 + r < src.plain_end(c, bk) && col < dv ? *reinterpret_cast<const float4*>(src_value(src, c, u0 + r) + col) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                }
            bar_sync(5, 512);
#pragma unroll 1
            for (uint32_t d = 0; d < 64; d += 4) {
                float4 q[4], k[4];
#pragma unroll
                for (int r = 0; r < 4; r++) q[r] = *reinterpret_cast<const float4*>(Qs + (4 * ty + r) * 64 + d);
#pragma unroll
                for (int i = 0; i < 4; i++) k[i] = *reinterpret_cast<const float4*>(Ks + (tx + 16 * i) * KP + d);
#pragma unroll
                for (int r = 0; r < 4; r++)
#pragma unroll
                    for (int i = 0; i < 4; i++) sc[r][i] = fmaf(q[r].w, k[i].w, fmaf(q[r].z, k[i].z, fmaf(q[r].y, k[i].y, fmaf(q[r].x, k[i].x, sc[r][i]))));
            }
        }
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const typename Src::Row w = src.query(c, 4 * ty + r);
            float mx = -INFINITY, sum = 0.0f;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                sc[r][i] = w.on ? src.slow_score(c, w, u0 + tx + 16 * i, sc[r][i]) : -INFINITY;
                mx = fmaxf(mx, sc[r][i]);
            }
            if (src.sigmoid()) {
#pragma unroll
                for (int i = 0; i < 4; i++) Ps[(4 * ty + r) * KP + tx + 16 * i] = sc[r][i] == -INFINITY ? 0.0f : ca_sigmoid(sc[r][i]);
                continue;
            }
#pragma unroll
            for (int x = 8; x > 0; x >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, x));
            const float mn = fmaxf(m[r], mx), al = m[r] == -INFINITY ? (mn == -INFINITY ? 1.0f : 0.0f) : expf(m[r] - mn);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float p = sc[r][i] == -INFINITY ? 0.0f : expf(sc[r][i] - mn);
                Ps[(4 * ty + r) * KP + tx + 16 * i] = p;
                sum += p;
            }
#pragma unroll
            for (int x = 8; x > 0; x >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x);
            l[r] = fmaf(l[r], al, sum);
            m[r] = mn;
#pragma unroll
            for (int k = 0; k < OC; k++) o[r][k] *= al;
        }
        bar_sync(5, 512);
#pragma unroll 1
        for (int j = 0; j < 64; j++) {
            float v[OC];
#pragma unroll
            for (int k = 0; k < OC; k++) v[k] = Vs[j * DV + tx + 16 * k];
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const float p = Ps[(4 * ty + r) * KP + j];
#pragma unroll
                for (int k = 0; k < OC; k++) if (p != 0.0f) o[r][k] = fmaf(p, v[k], o[r][k]);
            }
        }
    }
    bar_sync(5, 512);
    float* const out = sm;                             // [128][DV]
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const typename Src::Row w = src.query(c, 4 * ty + r);
        const float f = w.on ? src.finish(c, w, tx == 0, m[r], false, l[r], 1.0f) : 0.0f;
#pragma unroll
        for (int k = 0; k < OC; k++) out[(4 * ty + r) * DV + tx + 16 * k] = o[r][k] * f;
    }
    bar_sync(5, 512);
    for (uint32_t i = tid; i < c.nq * (DV / 4); i += 512) {
        const uint32_t r = i / (DV / 4), col = 4 * (i % (DV / 4));
        src.put(c, src.query(c, r), col, *reinterpret_cast<const float4*>(out + r * DV + col));
    }
}

// NC: 64-wide chunks of the key dimension; DV: value columns of the CTA (64 or 128)
template <class Src, int NC, int DV>
__global__ void __launch_bounds__(kAtcThreads, 1)
k_attention_tc(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const Src src, const AtcPlanes pl) {
    constexpr uint32_t BK = NC <= 2 ? 128 : 64, KC = BK / 64;       // keys per tile: scores twice, outputs and queries share the 512 columns of TMEM
    constexpr uint32_t kS = 0, kO = 2 * BK, kQ = kO + DV;           // TMEM columns; the CTA owns all 512, so their addresses are constants
    static_assert(kQ + 64 * NC <= 512, "TMEM columns");
    constexpr uint32_t kPieceK = BK * 128, kPieceV = DV * 128, kQPieces = 2 * NC;       // 128 rows of 64 NC f32 queries
    extern __shared__ uint8_t dsm_raw[];
    const uint32_t base = (smem_u32(dsm_raw) + 1023u) & ~1023u, bars = base + kAtcRing * kAtcPiece + kAtcShare + kAtcTiles * 12;
    const uint32_t full = bars, empty = full + 8 * kAtcRing, s_full = empty + 8 * kAtcRing, p_full = s_full + 16, o_full = p_full + 8, q_full = o_full + 8, tmem_slot = q_full + 8;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < kAtcRing; i++) { mbar_init(full + 8 * i, 1); mbar_init(empty + 8 * i, 1); }
        mbar_init(s_full, 1); mbar_init(s_full + 8, 1); mbar_init(p_full, 16); mbar_init(o_full, 1); mbar_init(q_full, 16);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 17) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(tmem_slot) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    uint32_t* const trouble = reinterpret_cast<uint32_t*>(dsm_raw + (tmem_slot + 4 - smem_u32(dsm_raw)));      // of the CTA: 1 rows that pairs cannot hold, 2 a wait that ran out
    if (threadIdx.x == 0) *trouble = 0;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const typename Src::Cta c = src.cta(BK);
    // class and scales of the first tiles: read from global memory inside the loop they cost every tile an L2 round trip
    float* const share = reinterpret_cast<float*>(dsm_raw + (base - smem_u32(dsm_raw)) + kAtcRing * kAtcPiece);
    float4* const ring = reinterpret_cast<float4*>(dsm_raw + (base - smem_u32(dsm_raw)));
    float2* const tile_inv = reinterpret_cast<float2*>(share + kAtcShare / 4);
    uint32_t* const tile_class = reinterpret_cast<uint32_t*>(tile_inv + kAtcTiles);
    const float* k_inv = pl.k_inv + (size_t)src.k_item(c) * pl.tiles;
    const float* v_inv = pl.v_inv + (size_t)src.v_item(c) * pl.tiles;
    for (uint32_t i = threadIdx.x; i < min(c.t1 - c.t0, kAtcTiles); i += kAtcThreads) {
        const uint32_t t = c.t0 + i;
        tile_class[i] = src.classify(c, t, BK);
        tile_inv[i] = make_float2(k_inv[t * BK / 128], v_inv[t * BK / 128]);
    }
    fence_before();
    __syncthreads();
    fence_after();
    auto class_of = [&](uint32_t t) { return t - c.t0 < kAtcTiles ? tile_class[t - c.t0] : src.classify(c, t, BK); };

    if (src.idle(c)) {                                               // uniform over the CTA
        if (threadIdx.x < 128) src.leave_empty(c, threadIdx.x);
    } else if (warp == 16) {
        if (lane == 0) {
            uint32_t slot = 0, phase = 1;                            // ring position
            bool ok = true;
            auto piece = [&](const CUtensorMap* map, uint32_t x, uint32_t y, uint32_t bytes) {
                if (ok) ok = mbar_wait(empty + 8 * slot, phase);
                if (ok && phase && slot == kAtcRing - kQPieces) ok = mbar_wait(q_full, 0);       // first time round: the queries are staged there
                if (!ok) return;
                mbar_expect_tx(full + 8 * slot, bytes);
                tma_2d(base + slot * kAtcPiece, map, x, y, full + 8 * slot);
                if (++slot == kAtcRing) { slot = 0; phase ^= 1; }
            };
            const uint32_t ky = src.k_item(c) * pl.tiles * 128, vy = src.v_item(c) * pl.vslice;
            auto values = [&](uint32_t t) {
                for (int part = 1; part >= 0; part--)                // lo first: the cross terms come first
                    for (uint32_t k = 0; k < KC; k++) piece(&map_v, part * pl.tiles * 128 + t * BK + 64 * k, vy, kPieceV);
            };
            uint32_t prev = 0;
            bool have = false;
            for (uint32_t t = c.t0; t < c.t1 && ok; t++) {
                if (!class_of(t)) continue;
                for (int part = 1; part >= 0; part--)
                    for (uint32_t k = 0; k < NC; k++) piece(&map_k, part * pl.dkp + 64 * k, ky + t * BK, kPieceK);
                if (have) values(prev);
                prev = t; have = true;
            }
            if (have) values(prev);
        }
        __syncwarp();
    } else if (warp == 17) {
        // The whole warp walks the tiles and waits; one elected lane issues.  Addresses stay warp-uniform that way: with the loop inside a
        // single lane's branch every MMA took 130 clocks to issue, twice what it takes to execute.
        constexpr uint32_t idesc_s = (1u << 4) | ((BK >> 3) << 17) | ((128u >> 4) << 24), idesc_o = (1u << 4) | ((DV >> 3) << 17) | ((128u >> 4) << 24);   // f16 x f16 -> f32
        const bool leader = elect_one();
        const uint32_t b0 = desc_low(base);
        uint32_t n_tiles = 0, slot = 0, phase = 0;                    // ring position
        for (uint32_t t = c.t0; t < c.t1; t++) n_tiles += class_of(t) ? 1 : 0;
        bool ok = mbar_wait(q_full, 0);
        fence_after();
        uint32_t held[4];                                             // ring slots of the hi pieces, which serve two products
        auto next = [&]() {                                           // the next piece has arrived
            const uint32_t s = slot;
            if (ok) ok = mbar_wait(full + 8 * s, phase);
            if (++slot == kAtcRing) { slot = 0; phase ^= 1; }
            return s;
        };
        // D += A B over the 64 keys or dims of ring slot s: A at TMEM column a, STEP columns from one 16 to the next
        auto product = [&](uint32_t d, uint32_t a, auto step, uint32_t s, uint32_t idesc, auto first) {
            const uint32_t b = b0 + s * (kAtcPiece >> 4);
            mma_ts<!decltype(first)::value>(d, a, b, idesc);
#pragma unroll
            for (uint32_t k = 1; k < 4; k++) mma_ts<true>(d, a + decltype(step)::value * k, b + 2 * k, idesc);
        };
        // three products of A (hi at a, lo at a + lo_at, `chunk` columns per piece) with N pieces of B: hi lo, lo hi, hi hi
        auto triple = [&](uint32_t d, uint32_t a, uint32_t lo_at, uint32_t chunk, auto step, auto count, uint32_t idesc) {
            constexpr uint32_t N = decltype(count)::value;
#pragma unroll
            for (uint32_t k = 0; k < N; k++) {
                const uint32_t s = next();
                fence_after();
                if (leader && ok) {
                    if (k == 0) product(d, a, step, s, idesc, std::true_type{}); else product(d, a + chunk * k, step, s, idesc, std::false_type{});
                    mma_commit(empty + 8 * s);
                }
            }
#pragma unroll
            for (uint32_t k = 0; k < N; k++) {
                held[k] = next();
                fence_after();
                if (leader && ok) product(d, a + lo_at + chunk * k, step, held[k], idesc, std::false_type{});
            }
            if (leader && ok) {
#pragma unroll
                for (uint32_t k = 0; k < N; k++) {
                    product(d, a + chunk * k, step, held[k], idesc, std::false_type{});
                    mma_commit(empty + 8 * held[k]);
                }
            }
        };
        auto scores = [&](uint32_t i) {
            triple(kS + (i & 1) * BK, kQ, 32 * NC, 32, std::integral_constant<uint32_t, 8>{}, std::integral_constant<uint32_t, NC>{}, idesc_s);
            if (leader && ok) mma_commit(s_full + 8 * (i & 1));
        };
        // probabilities of 16 keys lie in 16 columns: 8 with their hi pairs, 8 with their lo pairs
        auto values = [&](uint32_t i) {
            if (ok) ok = mbar_wait(p_full, i & 1);
            fence_after();
            triple(kO, kS + (i & 1) * BK, 8, 64, std::integral_constant<uint32_t, 16>{}, std::integral_constant<uint32_t, KC>{}, idesc_o);
            if (leader && ok) mma_commit(o_full);
        };
        for (uint32_t i = 0; i < n_tiles && ok; i++) {
            scores(i);
            if (i) values(i - 1);
        }
        if (n_tiles && ok) values(n_tiles - 1);
        __syncwarp();
    } else {
        // ── four threads per query row: quarter `part` of a tile's keys, of the output columns and of the query's dims ──
        constexpr int KW = BK / 4, OW = DV / 4;
        const uint32_t part = warp >> 2, row = (warp & 3) * 32 + lane, lanes = ((warp & 3) * 32) << 16;
        const typename Src::Row w = src.query(c, row);
        uint32_t n_share = 0;
        auto row_max = [&](float x) {                                // over the row's four threads; two buffers in turns, so one barrier is enough
            float* s = share + (n_share++ & 1) * 512;
            s[part * 128 + row] = x;
            bar_sync(1 + (warp & 3), 128);
            return fmaxf(fmaxf(s[row], s[128 + row]), fmaxf(s[256 + row], s[384 + row]));
        };
        // The queries come by whole rows (32 lanes, 512 contiguous bytes) into the ring's last pieces, which the loading warp leaves alone until
        // q_full, and a thread takes its quarter row from there: read from global memory row by thread they took 9000 clocks.
        float* const stage = share - (size_t)kQPieces * (kAtcPiece / 4);
        constexpr uint32_t Q4 = 16 * NC;                             // float4s of a row; float4 j of row r lies at place j ^ (r & 7)
        for (uint32_t i = threadIdx.x; i < 128 * Q4; i += 512) {
            const uint32_t r = i / Q4, j = i % Q4;
            const bool on = 4 * j < src.dk();
            const float* from = src.q_row(c, src.query(c, r)) + 4 * j;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(stage + 4 * (r * Q4 + (j ^ (r & 7))))), "l"(on ? from : from - 4 * j), "r"(on ? 16 : 0) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        bar_sync(5, 512);
        float q_inv, q_scale;
        bool wide;                                                    // the row's magnitudes lie too far apart
        {
            float4 x[4 * NC];                                        // 16 NC dims from 16 NC part on
            float mx = 0.0f;
#pragma unroll
            for (int i = 0; i < 4 * NC; i++) x[i] = *reinterpret_cast<const float4*>(stage + 4 * (row * Q4 + ((4 * NC * part + i) ^ (row & 7))));
#pragma unroll
            for (int i = 0; i < 4 * NC; i++) mx = abs_or_inf(abs_or_inf(abs_or_inf(abs_or_inf(mx, x[i].x), x[i].y), x[i].z), x[i].w);
            split_scale(row_max(mx), q_scale, q_inv);
            uint32_t small = 0;
#pragma unroll
            for (int i = 0; i < 4 * NC; i++) small += is_small(x[i].x, q_scale) + is_small(x[i].y, q_scale) + is_small(x[i].z, q_scale) + is_small(x[i].w, q_scale);
            wide = small >= kAtcSmallQuery;
#pragma unroll
            for (int i = 0; i < NC; i++) {                           // 16 dims: 8 columns of pairs
                uint32_t hi[8], lo[8];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    split2(x[4 * i + j].x * q_scale, x[4 * i + j].y * q_scale, hi[2 * j], lo[2 * j]);
                    split2(x[4 * i + j].z * q_scale, x[4 * i + j].w * q_scale, hi[2 * j + 1], lo[2 * j + 1]);
                }
                tmem_st(lanes + kQ + 8 * (NC * part + i), hi);
                tmem_st(lanes + kQ + 32 * NC + 8 * (NC * part + i), lo);
            }
            tmem_wait_st();
            fence_before();
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");       // the ring's last pieces are read: TMA may write them
            __syncwarp();
            if (lane == 0) mbar_arrive(q_full);
        }
        const float unit = src.scale(c) * kLog2e;
        const bool sigmoid = src.sigmoid();
        float o[OW];
#pragma unroll
        for (int i = 0; i < OW; i++) o[i] = 0.0f;
        float m = -INFINITY, l = 0.0f, alpha_prev = 1.0f, f_prev = 0.0f;
        bool ok = true, slow = wide || src.over(c) || !(q_inv == q_inv);
        uint32_t it = 0;
        auto add_output = [&](uint32_t i) {                          // outputs of tile i join the running ones
            if (ok) ok = __all_sync(0xffffffffu, mbar_wait(o_full, i & 1));
            fence_after();
            uint32_t v[OW];
            tmem_ld(lanes + kO + OW * part, v);
            tmem_wait_ld(v);
#pragma unroll
            for (int j = 0; j < OW; j += 2) {
                const float2 r = __ffma2_rn(make_float2(o[j], o[j + 1]), make_float2(alpha_prev, alpha_prev),
                                            __fmul2_rn(make_float2(__uint_as_float(v[j]), __uint_as_float(v[j + 1])), make_float2(f_prev, f_prev)));
                o[j] = r.x; o[j + 1] = r.y;
            }
        };
        for (uint32_t t = c.t0; t < c.t1; t++) {
            const uint32_t cls = class_of(t);
            if (!cls) continue;
            const float2 inv = t - c.t0 < kAtcTiles ? tile_inv[t - c.t0] : make_float2(k_inv[t * BK / 128], v_inv[t * BK / 128]);
            const float f = q_inv * inv.x * unit;
            slow = slow || !(fabsf(f) < kAtcBig) || !(inv.y < kAtcBig);
            const bool plain = src.plain_tile() && cls == 1;
            if (ok) ok = __all_sync(0xffffffffu, mbar_wait(s_full + 8 * (it & 1), (it >> 1) & 1));
            fence_after();
            const uint32_t s = lanes + kS + (it & 1) * BK + KW * part, u0 = t * BK + KW * part;
            uint32_t v[KW];
            tmem_ld(s, v);
            tmem_wait_ld(v);
            float x[KW], alpha = 1.0f, shift = 14.0f;                // scores in units of log2; probabilities times 2^14
#pragma unroll
            for (int j = 0; j < KW; j++) x[j] = __uint_as_float(v[j]) * f;
            if (!plain) src.scores(c, w, t, u0, cls, x);
            if (!sigmoid) {
                float m0 = x[0], m1 = x[1];
#pragma unroll
                for (int j = 2; j < KW; j += 2) { m0 = fmaxf(m0, x[j]); m1 = fmaxf(m1, x[j + 1]); }
                const float mx = row_max(fmaxf(m0, m1)), m_new = fmaxf(m, mx);
                slow = slow || mx == INFINITY;
                alpha = m == -INFINITY ? 0.0f : ex2(m - m_new);
                m = m_new;
                if (m_new != -INFINITY) shift -= m_new;
#pragma unroll
                for (int j = 0; j < KW; j++) x[j] = ex2(x[j] + shift);
            } else {
#pragma unroll
                for (int j = 0; j < KW; j++) x[j] = x[j] == -INFINITY ? 0.0f : kPScale * ca_sigmoid(x[j] * kLn2);
            }
            float l0 = 0.0f, l1 = 0.0f;
#pragma unroll
            for (int j = 0; j < KW; j += 2) {
                l0 += x[j]; l1 += x[j + 1];
                split2(x[j], x[j + 1], v[(j / 16) * 16 + (j % 16) / 2], v[(j / 16) * 16 + 8 + (j % 16) / 2]);
            }
            tmem_st(s, v);
            l = fmaf(l, alpha, l0 + l1);
            tmem_wait_st();
            if (it) add_output(it - 1);
            alpha_prev = alpha; f_prev = inv.y;
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_full);
            it++;
        }
        if (it) add_output(it - 1);
        {
            float* s = share + (n_share & 1) * 512;                  // the row's sum
            s[part * 128 + row] = l;
            bar_sync(1 + (warp & 3), 128);
            l = (s[row] + s[128 + row]) + (s[256 + row] + s[384 + row]);
        }
        // Outputs leave by whole rows too, through the idle ring.
        auto place = [&](int j) { return row * (DV / 4) + (((OW * part + j) / 4) ^ (row & 7)); };
        const float f = w.on ? src.finish(c, w, part == 0, m, true, l, kPInv) : 0.0f;
#pragma unroll
        for (int j = 0; j < OW; j += 4) ring[place(j)] = make_float4(o[j] * f, o[j + 1] * f, o[j + 2] * f, o[j + 3] * f);
        if (slow || (m < kAtcLow && m != -INFINITY)) atomicOr(trouble, 1u);
        if (!ok) { atomicOr(trouble, 2u); if (lane == 0) count_timeout(); }
        bar_sync(5, 512);
        const uint32_t what = *trouble;
        const bool lost = what & 2;                                  // (what still arrives in the ring is not looked at)
        if (what == 1) atc_plain<DV>(src, c, BK, reinterpret_cast<float*>(ring));
        else
        for (uint32_t i = threadIdx.x; i < c.nq * (DV / 4); i += 512) {
            const uint32_t r = i / (DV / 4), j = i % (DV / 4);
            src.put(c, src.query(c, r), 4 * j, lost ? make_float4(kNotANumber, kNotANumber, kNotANumber, kNotANumber) : ring[r * (DV / 4) + (j ^ (r & 7))]);
        }
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    __syncwarp();
    fence_before();
    __syncthreads();
    if (warp == 17) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(0u) : "memory");
}

bool encode_plane(CUtensorMap* map, void* p, uint64_t width, uint64_t rows, uint32_t box_rows) {
    const cuuint64_t dims[2] = {width, rows}, stride[1] = {width * 2};
    const cuuint32_t box[2] = {64, box_rows}, one[2] = {1, 1};
    EncodeTiledFn fn = encode_tiled();
    if (!fn) { zg_set_error("cuTensorMapEncodeTiled entry point not available"); return false; }
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, p, dims, stride, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { zg_set_error("cuTensorMapEncodeTiled(attention planes) failed (%d)", (int)r); return false; }
    return true;
}
size_t up64(size_t n) { return (n + 63) & ~(size_t)63; }
// scratch: planes, then scales, then whatever the caller adds; offsets in f32 slots
struct AtcLayout { size_t k, v, k_inv, v_inv, total; };
AtcLayout layout(const AtcPlanes& p) {
    AtcLayout L;
    size_t o = 0;
    L.k = o; o += up64((size_t)p.k_items * p.tiles * 128 * p.dkp);
    L.v = o; o += up64((size_t)p.v_items * p.vslice * p.tiles * 128);
    L.k_inv = o; o += up64((size_t)p.k_items * p.tiles);
    L.v_inv = o; o += up64((size_t)p.v_items * p.tiles);
    L.total = o;
    return L;
}
void place(AtcPlanes& p, float* scratch) {
    const AtcLayout L = layout(p);
    p.k = reinterpret_cast<__half*>(scratch + L.k); p.v = reinterpret_cast<__half*>(scratch + L.v);
    p.k_inv = scratch + L.k_inv; p.v_inv = scratch + L.v_inv;
}
template <class Src, int NC, int DV>
bool launch(const Src& src, const AtcPlanes& pl, dim3 grid, cudaStream_t st) {
    constexpr uint32_t BK = NC <= 2 ? 128 : 64;
    constexpr int C = NC > DV / 64 ? NC : DV / 64;
    CUtensorMap mk, mv;
    if (!encode_plane(&mk, pl.k, 2 * pl.dkp, (uint64_t)pl.k_items * pl.tiles * 128, BK) || !encode_plane(&mv, pl.v, (uint64_t)2 * pl.tiles * 128, (uint64_t)pl.v_items * pl.vslice, DV)) return false;
    if (!zg_smem_limit<k_attention_tc<Src, NC, DV>>(kAtcSmem)) return false;
    const uint32_t items = pl.k_items + pl.v_items, per_item = (4 * zg_sm_count() + items - 1) / items;
    launch_pdl(k_atc_prep<Src, C>, dim3(pl.tiles < per_item ? pl.tiles : per_item, items), dim3(kPrepThreads), 0, st, src, pl);
    ZG_COUNT_LAUNCH();
    launch_pdl(k_attention_tc<Src, NC, DV>, grid, dim3(kAtcThreads), kAtcSmem, st, mk, mv, src, pl);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { zg_set_error("attention launch failed: %s", cudaGetErrorString(e)); return false; }
    ZG_COUNT_LAUNCH();
    return true;
}
template <class Src>
bool launch_dims(const Src& src, const AtcPlanes& pl, dim3 grid, cudaStream_t st) {
    const uint32_t nc = pl.dkp / 64;
#define ZG_ATC(NC_) (pl.vslice == 64 ? launch<Src, NC_, 64>(src, pl, grid, st) : launch<Src, NC_, 128>(src, pl, grid, st))
    return nc == 1 ? ZG_ATC(1) : nc == 2 ? ZG_ATC(2) : nc == 3 ? ZG_ATC(3) : ZG_ATC(4);
#undef ZG_ATC
}
struct CachedPlan { AtcPlanes pl; uint32_t rh, row_tiles, splits; };
CachedPlan cached_plan(const ZgAtcShape& s, int n_sm) {
    CachedPlan P = {};
    P.pl.vslice = s.dv <= 64 ? 64 : 128; P.pl.n_vs = (s.dv + P.pl.vslice - 1) / P.pl.vslice;
    P.pl.dk = s.dk; P.pl.dv = s.dv; P.pl.dkp = (s.dk + 63) / 64 * 64;
    P.pl.k_items = s.G * s.maps; P.pl.v_items = s.G * P.pl.n_vs; P.pl.tiles = (s.reach + 127) / 128;
    P.rh = s.H / s.G; P.row_tiles = (s.T * P.rh + 127) / 128;
    // few row tiles over many keys: key ranges of at least two tiles of 128 go to CTAs of their own until the SMs are covered
    const uint32_t ctas = P.row_tiles * P.pl.k_items * P.pl.n_vs;
    uint32_t S = (uint32_t)n_sm / (ctas ? ctas : 1), most = P.pl.tiles / 2;
    if (S > most) S = most;
    P.splits = S < 2 ? 1 : S > 64 ? 64 : S;
    return P;
}
}  // namespace

// Measured against the SIMT kernels over 32 shapes (16 to 1024 tokens, 1 to 16 heads of 32 to 160, windows of 71 to 749 and whole caches): with
// tokens x heads x keys x (dk + dv) of 60 M and more this form was 1.0 to 2.7 times as fast, 11.9 times at 1024 tokens x 16 heads x 2048 keys of
// 128; between 5 M and 36 M it took 0.8 to 1.1 times as long: the split of the cache and the start of the pipeline cost about 10 us.
// `keys` of a causal mask is the cache's capacity, since the position is known on the device only.  16 heads over 4 of 128, capacity 4096, SIMT / this form: 16 tokens at
// position 0 27 / 28 us, at 500 42 / 30; 64 tokens at 0 29 / 35, at 1000 74 / 37; 256 tokens at 0 51 / 53, at 2000 291 / 68: only the first step of a sequence loses.
bool zg_attention_tc_usable(const ZgAtcShape& s) {
    return s.dk >= 32 && s.dk <= 256 && s.dv >= 32 && s.T >= 16 && (uint64_t)s.T * s.H * s.maps * s.keys * (s.dk + s.dv) >= 48000000ull;
}
size_t zg_attention_tc_scratch_elems(const ZgAtcShape& s, int n_sm) {
    const CachedPlan P = cached_plan(s, n_sm);
    return layout(P.pl).total + (P.splits > 1 ? (size_t)s.T * s.H * s.maps * P.splits * (4 + s.dv) : 0);
}
bool zg_attention_tc_launch(const ZgAtcShape& s, const void* args, float* scratch, int n_sm, cudaStream_t st, uint32_t* splits, float** part) {
    const CaArgs& a = *static_cast<const CaArgs*>(args);
    CachedPlan P = cached_plan(s, n_sm);
    place(P.pl, scratch);
    *splits = P.splits;
    *part = P.splits > 1 ? scratch + layout(P.pl).total : nullptr;
    const dim3 grid(P.row_tiles * P.pl.k_items * P.pl.n_vs, P.splits);
    if (a.cap > 0.0f || a.tab || a.wkind || a.pool) {
        AtcCached<true> src = {a, P.rh, P.row_tiles, P.pl.n_vs, P.pl.vslice, P.splits, P.pl.tiles, *part};
        return launch_dims(src, P.pl, grid, st);
    }
    AtcCached<false> src = {a, P.rh, P.row_tiles, P.pl.n_vs, P.pl.vslice, P.splits, P.pl.tiles, *part};
    return launch_dims(src, P.pl, grid, st);
}

// ── DeviceOp.attention batches ──
// Keys that planes are laid out for: those up to the next head, layer or operand in the same buffer (a head's rows may lie between other heads' rows; what
// starts past the rows it attends over now ends them), and inside its key, value and mask operands.  An op that is refreshed to more is evaluated in plain f32.
static size_t attention_key_bound(const ZgOp& op, const size_t* elems, const std::map<uint32_t, std::vector<size_t>>& starts) {
    const auto& a = op.u.attention;
    const size_t now = std::max(a.seq_kv, a.seq_q);
    auto rows = [](size_t n, size_t off, size_t width, size_t stride) { return n < off + width ? (size_t)0 : stride ? (n - off - width) / stride + 1 : (size_t)UINT32_MAX; };
    auto slab = [&](uint32_t buf, size_t off, size_t stride) {
        const std::vector<size_t>& at = starts.at(buf);
        const auto next = std::lower_bound(at.begin(), at.end(), off + (now ? now - 1 : 0) * stride + a.d_head);
        return rows(next == at.end() ? elems[buf] : std::min(elems[buf], *next), off, a.d_head, stride);
    };
    size_t n = std::min(slab(a.k, a.k_off, a.k_cs), slab(a.v, a.v_off, a.v_cs));
    if (a.has_mask) n = std::min(n, rows(elems[a.mask], (size_t)a.mask_off + (size_t)(a.seq_q - 1) * a.mask_cs, 1, a.mask_rs));
    return n;
}
bool zg_atc_program_plan(const std::vector<ZgOp>& all, const ZgOp* const* ops, uint32_t count, const size_t* buffer_elems, ZgAtcPlan* plan) {
    const auto& first = ops[0]->u.attention;
    size_t keys = 0, now = 0;
    std::map<uint32_t, std::vector<size_t>> starts;                   // where keys and values of the program's attentions start in a buffer
    for (const ZgOp& op : all)
        if (op.tag == ZG_OP_ATTENTION) { starts[op.u.attention.k].push_back(op.u.attention.k_off); starts[op.u.attention.v].push_back(op.u.attention.v_off); }
    for (auto& b : starts) std::sort(b.second.begin(), b.second.end());
    std::map<uint32_t, size_t> operands;
    std::map<std::vector<uint32_t>, uint32_t> kv, masks;
    std::vector<uint32_t> kv_rep, mask_rep;
    plan->map.assign(2 * (size_t)count, 0);
    for (uint32_t i = 0; i < count; i++) {
        const auto& a = ops[i]->u.attention;
        keys = std::max(keys, attention_key_bound(*ops[i], buffer_elems, starts));
        now = std::max(now, (size_t)a.seq_kv);
        operands[a.k] = buffer_elems[a.k]; operands[a.v] = buffer_elems[a.v];
        const auto k = kv.emplace(std::vector<uint32_t>{a.k, a.k_off, a.k_cs, a.v, a.v_off, a.v_cs}, (uint32_t)kv.size());
        if (k.second) kv_rep.push_back(i);
        plan->map[i] = k.first->second;
        if (!a.has_mask) continue;
        const auto m = masks.emplace(std::vector<uint32_t>{a.mask, a.mask_off, a.mask_rs, a.mask_cs}, (uint32_t)masks.size());
        if (m.second) mask_rep.push_back(i);
        plan->map[count + i] = m.first->second;
    }
    // a head that reads on into something else's rows: no more than twice what the operands hold
    size_t most = 0;
    for (const auto& b : operands) most += 2 * b.second;
    most = most / (2 * (size_t)first.d_head * 128 * kv.size()) * 128;
    keys = std::min(keys, std::max(most, (size_t)128));
    if (keys == 0 || keys < now || keys > kAtcProgramKeys) return false;
    plan->map.insert(plan->map.end(), kv_rep.begin(), kv_rep.end());
    plan->map.insert(plan->map.end(), mask_rep.begin(), mask_rep.end());
    plan->count = count; plan->kv_items = (uint32_t)kv_rep.size(); plan->mask_items = (uint32_t)mask_rep.size();
    plan->seq_q = first.seq_q; plan->head = first.d_head; plan->tiles = (uint32_t)((keys + 127) / 128);
    return true;
}
static AtcPlanes program_planes(const ZgAtcPlan& p) {
    AtcPlanes pl = {};
    pl.dkp = pl.vslice = pl.dk = pl.dv = p.head;
    pl.k_items = pl.v_items = p.kv_items; pl.n_vs = 1; pl.tiles = p.tiles;
    return pl;
}
static size_t mask_tiles(const ZgAtcPlan& p) { return (size_t)p.mask_items * ((p.seq_q + 127) / 128) * p.tiles; }
size_t zg_atc_program_scratch_elems(const ZgAtcPlan& p) { return layout(program_planes(p)).total + mask_tiles(p) * 512 + (mask_tiles(p) + 3) / 4; }
bool zg_atc_program_launch(const ZgAtcPlan& p, const ZgBatchEntry* d_entries, const uint32_t* d_map, const uint32_t* d_dyn, float* scratch, cudaStream_t st) {
    AtcPlanes pl = program_planes(p);
    place(pl, scratch);
    const uint32_t row_tiles = (p.seq_q + 127) / 128;
    AtcProgram src = {d_entries, d_dyn, d_map, p.count, p.kv_items, p.mask_items, p.seq_q, p.head, row_tiles, p.tiles, nullptr, nullptr};
    src.bits = reinterpret_cast<uint32_t*>(scratch + layout(pl).total);
    src.classes = reinterpret_cast<uint8_t*>(src.bits + mask_tiles(p) * 512);
    if (p.mask_items) {
        launch_pdl(k_atc_masks, dim3(p.tiles, row_tiles, p.mask_items), dim3(512), 0, st, src);
        ZG_COUNT_LAUNCH();
    }
    const dim3 grid(row_tiles * p.count);
    return p.head == 64 ? launch<AtcProgram, 1, 64>(src, pl, grid, st) : launch<AtcProgram, 2, 128>(src, pl, grid, st);
}
unsigned int zg_attention_tc_timeouts() { return tc_timeouts(); }
