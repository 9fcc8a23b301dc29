"""CACHED_ATTENTION with many rows (the tensor-core form: f32 operands split into half-precision pairs) in two-op programs against float64:
key dimensions and value widths around the 64-wide chunks, partial row and key tiles, every mask, ring wrap-around and a second state slot, caps, score
tables, sinks, sigmoid weights, several maps, key ranges dealt to several CTAs, magnitudes far from 1, and rows that hold a NaN or an infinity.

Tolerance: a split operand keeps its value to 2^-23 of itself or 2^-39 of its row's (tile's) largest, and f32 sums of up to a thousand terms add a few
2^-24 of the largest partial sum: 1e-5 of the output's scale is ten times what scores up to about 10 make of that."""
import numpy as np
import pytest

from test_gpu_recops import ctl_words, run
from test_gpu_split_gemm import waits_given_up

pytestmark = pytest.mark.gpu


def reference(q, keys, vals, seen, scale, cap=0.0, table=None, dist=None, sink=None, sigmoid=False):
    """One head: q [T, dk], keys [n, dk], vals [n, dv], seen [T, n]."""
    s = q @ keys.T * scale
    if cap:
        s = cap * np.tanh(s / cap)
    if table is not None:
        s = s + table[np.clip(dist, 0, len(table) - 1)]
    if sigmoid:
        return np.where(seen, 1.0 / (1.0 + np.exp(-s)), 0.0) @ vals
    s = np.where(seen, s, -np.inf)
    m = s.max(1, keepdims=True)
    e = np.exp(s - m)
    return e @ vals / (e.sum(1, keepdims=True) + (np.exp(sink - m) if sink is not None else 0.0))


def case(be, T, pos, H, G, dk, dv, maps=1, mask="causal", size=0, R=None, slot=0, cap=0.0, table=False, sink=False, sigmoid=False, out_scale=None, gain=1.0, seed=0, poison=None, block=0):
    from zgml_b200 import DeviceBuffer, DeviceOp, ExternBuffer, abi
    r = np.random.default_rng(seed)
    kw, vw = G * maps * dk, G * dv
    R = R or pos + T
    kc, vc = (gain * r.standard_normal((2, R, kw))).astype(np.float32), r.standard_normal((2, R, vw)).astype(np.float32) * np.float32(gain)
    if poison:
        poison(kc[slot], vc[slot])
    q = (r.standard_normal((T, H * maps * dk)) * 2.0 / gain).astype(np.float32)
    bk, bv = DeviceBuffer(be, kc.nbytes, zero=False), DeviceBuffer(be, vc.nbytes, zero=False)
    bk.upload(kc)
    bv.upload(vc)
    sizes, ext, io, kwargs = [T * H * maps * dv, q.size, bk.elems, bv.elems, 8 + T], [ExternBuffer(2, bk), ExternBuffer(3, bv)], [(1, q), (4, ctl_words(pos, slot))], {}
    tab = (r.standard_normal((H * maps, R)) * 0.5).astype(np.float32) if table else None
    if table:
        sizes.append(tab.size)
        io.append((len(sizes) - 1, tab))
        kwargs.update(score_table=len(sizes) - 1, table_len=R)
    sk = r.standard_normal(H * maps).astype(np.float32) if sink else None
    if sink:
        sizes.append(sk.size)
        io.append((len(sizes) - 1, sk))
        kwargs.update(sink=len(sizes) - 1, sink_wdt=abi.W_F32)
    op = DeviceOp.cached_attention(0, 1, 2, 3, 4, 0, 0, 0, T, H, G, maps, dk, dv, H * maps * dk, kw, vw, R, dk ** -0.5, mask=mask, mask_size=size, softcap=cap,
                                   weights="sigmoid" if sigmoid else "softmax", out_scale=out_scale, **kwargs)
    got = run(be, [op], sizes, io, 0, (T, H, maps, dv), ext)
    bk.free()
    bv.free()
    p = np.arange(pos, pos + T)
    lo = {"causal": 0 * p, "window": np.maximum(p + 1 - size, 0), "block": p - p % max(size, 1)}[mask]
    j = np.arange(lo[0], pos + T)
    seen, dist = (j <= p[:, None]) & (j >= lo[:, None]), p[:, None] - j
    want = np.empty((T, H, maps, dv))
    for h in range(H):
        g = h // (H // G)
        for m in range(maps):
            keys, vals = kc[slot][j % R][:, (g * maps + m) * dk:(g * maps + m + 1) * dk].astype(np.float64), vc[slot][j % R][:, g * dv:(g + 1) * dv].astype(np.float64)
            with np.errstate(invalid="ignore"):
                want[:, h, m] = reference(q[:, (h * maps + m) * dk:(h * maps + m + 1) * dk].astype(np.float64), keys, vals, seen, dk ** -0.5, cap, tab[h * maps + m] if table else None,
                                          dist, sk[h * maps + m] if sink else None, sigmoid) * (out_scale or 1.0)
    return got, want, seen, j


def close(got, want):
    return np.abs(got - want).max() <= 1e-5 * np.abs(want).max()


@pytest.mark.parametrize("shape", [
    dict(T=257, pos=0, H=8, G=8, dk=64, dv=64), dict(T=200, pos=131, H=8, G=2, dk=128, dv=128, sink=True), dict(T=130, pos=300, H=16, G=4, dk=36, dv=100),
    dict(T=129, pos=127, H=12, G=4, dk=160, dv=128, out_scale=0.5), dict(T=96, pos=500, H=8, G=1, dk=192, dv=128), dict(T=64, pos=900, H=8, G=2, dk=256, dv=200, sink=True),
    dict(T=16, pos=4000, H=8, G=8, dk=128, dv=128), dict(T=385, pos=77, H=8, G=4, dk=96, dv=64, mask="window", size=190, R=600), dict(T=300, pos=1000, H=8, G=8, dk=64, dv=32, mask="window", size=333, R=640),
    dict(T=300, pos=650, H=8, G=4, dk=64, dv=64, mask="block", size=400, R=800, slot=1), dict(T=150, pos=100, H=8, G=4, dk=64, dv=128, maps=2, cap=3.0, table=True),
    dict(T=260, pos=60, H=8, G=4, dk=128, dv=64, table=True, sigmoid=True), dict(T=200, pos=333, H=8, G=4, dk=192, dv=64, cap=2.0, sink=True, slot=1),
    dict(T=200, pos=100, H=8, G=4, dk=128, dv=128, gain=1e-12), dict(T=200, pos=100, H=8, G=4, dk=128, dv=128, gain=1e15)])
def test_many_rows(cuda_backend, shape):
    got, want, _, _ = case(cuda_backend, **shape)
    assert close(got, want)


@pytest.mark.parametrize("shape", [
    dict(T=16, pos=0, H=8, G=8, dk=64, dv=64, R=8192), dict(T=16, pos=300, H=8, G=8, dk=64, dv=128, R=8192, sink=True), dict(T=17, pos=2000, H=8, G=4, dk=160, dv=64, R=8000, sigmoid=True),
    dict(T=300, pos=0, H=8, G=2, dk=64, dv=64, R=20000), dict(T=1, pos=0, H=16, G=1, dk=64, dv=64, R=6000), dict(T=1, pos=30, H=16, G=1, dk=320, dv=256, R=6000, sink=True),
    dict(T=1, pos=2047, H=8, G=1, dk=128, dv=128, R=6000), dict(T=2, pos=2048, H=8, G=1, dk=128, dv=64, R=6000, sigmoid=True), dict(T=1, pos=4735, H=4, G=1, dk=64, dv=64, R=6000, out_scale=0.5),
    dict(T=1, pos=5999, H=16, G=1, dk=64, dv=64, R=6000), dict(T=1, pos=900, H=4, G=1, dk=64, dv=64, R=6000, mask="block", size=1000, slot=1)],
    ids=lambda d: " ".join(f"{k}{v}" for k, v in d.items() if k in ("T", "pos", "dk", "R")))
def test_steps_shorter_than_their_cache(cuda_backend, shape):
    """Key shares are planned for the cache's capacity and dealt by what a step sees: records of shares that are not used hold anything."""
    got, want, _, _ = case(cuda_backend, **shape)
    assert close(got, want)


def direct(be, q, k, v, pos, H, G, d):
    """Causal CACHED_ATTENTION of rows q [T, H d] over the cache rows k, v [pos + T, G d]."""
    from zgml_b200 import DeviceBuffer, DeviceOp, ExternBuffer
    T = len(q)
    q, k, v = (np.ascontiguousarray(a, np.float32) for a in (q, k, v))
    bk, bv = DeviceBuffer(be, k.nbytes, zero=False), DeviceBuffer(be, v.nbytes, zero=False)
    bk.upload(k)
    bv.upload(v)
    op = DeviceOp.cached_attention(0, 1, 2, 3, 4, 0, 0, 0, T, H, G, 1, d, d, H * d, G * d, G * d, pos + T, d ** -0.5, mask="causal")
    got = run(be, [op], [T * H * d, q.size, bk.elems, bv.elems, 8 + T], [(1, q), (4, ctl_words(pos, 0))], 0, (T, H, d), [ExternBuffer(2, bk), ExternBuffer(3, bv)])
    bk.free()
    bv.free()
    seen = np.arange(pos + T) <= np.arange(pos, pos + T)[:, None]
    part = lambda a, i: a[:, i * d:(i + 1) * d].astype(np.float64)
    return got, np.stack([reference(part(q, h), part(k, h * G // H), part(v, h * G // H), seen, d ** -0.5) for h in range(H)], 1)


@pytest.mark.parametrize("what", ["key", "value", "column", "dims"])
def test_magnitudes_far_apart_within_a_tile(cuda_backend, what):
    """A large key or value that only the last rows see, a value column far below the others, and queries and keys whose large dims meet zeros: what is small keeps
    its bits, column by column."""
    r = np.random.default_rng(12)
    T, pos, H, G, d = 200, 120, 8, 4, 128
    k, v, q = r.standard_normal((pos + T, G * d)), r.standard_normal((pos + T, G * d)), r.standard_normal((T, H * d))
    if what == "key":
        k[300] *= 2.0 ** 24
    elif what == "value":
        v[300] *= 2.0 ** 24
    elif what == "column":
        v[:, 5::d] *= 2.0 ** -24
    else:
        k[:, 0::d], k[:, 1::d], q[:, 0::d], q[:, 1::d] = 2.0 ** 22, 0.0, 0.0, 2.0 ** 22
    got, want = direct(cuda_backend, q, k, v, pos, H, G, d)
    rows = slice(0, 300 - pos)                                         # those that do not see position 300
    assert (np.abs(got - want)[rows].max((0, 1)) <= 1e-5 * np.abs(want)[rows].max((0, 1))).all()
    assert np.isfinite(got).all()


@pytest.mark.parametrize("what", ["values", "orthogonal"])
def test_magnitudes_near_the_largest_float(cuda_backend, what):
    """Values of 1e35 are averaged; queries of 1e24 meet keys of 1e24 in other dims (every score is a plain 0) and ordinary ones in none."""
    r = np.random.default_rng(11)
    T, pos, H, G, d = 200, 100, 8, 4, 128
    k, v, q = r.standard_normal((pos + T, G * d)), r.standard_normal((pos + T, G * d)), r.standard_normal((T, H * d))
    if what == "values":
        v *= 1e35
    else:
        k.reshape(pos + T, G, d)[:, :, :64] = 0.0
        q.reshape(T, H, d)[:, :, 64:] = 0.0
        k, q = k * 1e24, q * 1e24
    got, want = direct(cuda_backend, q, k, v, pos, H, G, d)
    assert close(got, want)


@pytest.mark.parametrize("what", ["nan key", "nan value", "infinite value"])
def test_rows_that_see_nothing_non_finite_are_exact(cuda_backend, what):
    """Position 150 of every key head or value head is poisoned: the queries before it are as they were, and those that see it are not finite."""
    def poison(k, v):
        (k if what == "nan key" else v)[150] = np.inf if what == "infinite value" else np.nan
    got, _, seen, j = case(cuda_backend, T=200, pos=60, H=8, G=4, dk=128, dv=128, poison=poison, seed=3)
    clean, want, _, _ = case(cuda_backend, T=200, pos=60, H=8, G=4, dk=128, dv=128, seed=3)
    sees = seen[:, j == 150][:, 0]
    assert close(clean, want) and close(got[~sees], want[~sees])
    assert not np.isfinite(got[sees]).any()


def test_batched_heads_with_their_own_masks_and_a_refreshed_length(cuda_backend):
    """DeviceOp.attention of a prompt: five heads over two key / value slabs and three masks — zeros and -inf, additive values, one laid out query-contiguous — and
    none; then the same compiled program over fewer keys."""
    import ctypes as C
    from zgml_b200 import DeviceOp, DeviceProgram, ProgramIO
    r = np.random.default_rng(5)
    T, S, dh, H = 141, 300, 64, 5
    q, k, v = r.standard_normal((H, T, dh)).astype(np.float32), r.standard_normal((2, S, dh)).astype(np.float32), r.standard_normal((2, S, dh)).astype(np.float32)
    m0 = np.where(r.random((T, S)) < 0.4, -np.inf, 0.0).astype(np.float32)
    m0[:, 128:256] = -np.inf                                          # a whole tile nobody sees, beside tiles that every row sees in part
    m1 = np.where(r.random((T, S)) < 0.2, -np.inf, r.standard_normal((T, S))).astype(np.float32)
    m0[7], m1[7] = -np.inf, -np.inf                                   # a row that sees nothing: zeros
    masks = [m0, m1, m1, m0, None]
    mask_buf = np.concatenate([m0.ravel(), m1.ravel(), m1.T.ravel()]).astype(np.float32)
    geom = [(0, 1, S), (T * S, 1, S), (2 * T * S, T, 1), (0, 1, S), (0, 1, S)]                 # offset, stride between keys, between queries
    ops = [DeviceOp.attention(4, 0, 1, 2, 3, masks[h] is not None, dh, T, 270, 0.3, h * T * dh, h % 2 * S * dh, h % 2 * S * dh, geom[h][0], h * T * dh, 1, dh, 1, dh, 1, dh, geom[h][1],
                              geom[h][2], 1, dh) for h in range(H)]
    prog = DeviceProgram(ops, [q.size, k.size, v.size, mask_buf.size, q.size], [], [])
    handle = cuda_backend.compile_program(prog)
    ins = [ProgramIO(i, a.ravel()) for i, a in enumerate((q, k, v, mask_buf))]
    for n in (270, 129, 300):
        for o in ops:
            o.u.attention.seq_kv = n
        cuda_backend.refresh_program(handle, ops)
        got = np.zeros((H, T, dh), np.float32)
        cuda_backend.execute_program(handle, ins, [ProgramIO(4, got)])
        for h in range(H):
            s = q[h].astype(np.float64) @ k[h % 2, :n].astype(np.float64).T * 0.3 + (0.0 if masks[h] is None else masks[h][:, :n].astype(np.float64))
            top = s.max(1, keepdims=True)
            e = np.exp(s - np.where(np.isfinite(top), top, 0.0))
            want = e @ v[h % 2, :n].astype(np.float64) / np.maximum(e.sum(1, keepdims=True), 1e-300)
            assert close(got[h], want), (n, h)
    cuda_backend.free_program(handle)


@pytest.mark.parametrize("shape", [
    dict(T=200, pos=1500, H=8, G=4, dk=128, dv=128, size=300, pool=7), dict(T=64, pos=3000, H=8, G=2, dk=192, dv=64, size=100, pool=3, cap=4.0),
    dict(T=16, pos=6000, H=8, G=8, dk=128, dv=128, size=200, pool=4, sink=True), dict(T=130, pos=0, H=16, G=4, dk=64, dv=100, size=64, pool=1, sink=True, cap=3.0),
    dict(T=150, pos=1024, H=8, G=8, dk=96, dv=64, size=513, pool=5), dict(T=200, pos=1500, H=8, G=4, dk=128, dv=128, size=300, pool=7, bad="key"),
    dict(T=200, pos=1500, H=8, G=4, dk=128, dv=128, size=300, pool=7, bad="value")], ids=lambda d: " ".join(f"{k}{v}" for k, v in d.items() if k in ("T", "pos", "dk", "pool", "bad")))
def test_pooled_blocks_of_many_rows(cuda_backend, shape):
    """Mask "pooled": block means and window positions that share a key tile, a ring that wraps, the second slot, key shares, 64-key tiles; a block that holds no
    number leaves the rows that do not see it exact."""
    from zgml_b200 import DeviceBuffer, DeviceOp, ExternBuffer, abi
    T, pos, H, G, dk, dv, size, pool = (shape[k] for k in ("T", "pos", "H", "G", "dk", "dv", "size", "pool"))
    cap, bad = shape.get("cap", 0.0), shape.get("bad")
    r = np.random.default_rng(T + pos)
    n, width, R = pos + T, G * (dk + dv), size - 1 + T + 5
    NB = n // pool
    kv = r.standard_normal((n, width)).astype(np.float32)
    means = kv[:NB * pool].astype(np.float64).reshape(NB, pool, width).mean(1).astype(np.float32) * np.float32(pool ** 0.5)
    broken = (pos + T // 2 - size) // pool                             # seen from the middle of the step on
    sees = np.arange(pos, n) + 1 - size >= (broken + 1) * pool
    if bad:
        means[broken, slice(0, G * dk) if bad == "key" else slice(G * dk, width)] = np.nan
    cache, pooled = np.zeros((2, R, width), np.float32), np.zeros((2, NB, width), np.float32)
    last = np.arange(max(0, n - R), n)
    cache[1][last % R] = kv[last]
    pooled[1] = means
    bc, bp = DeviceBuffer(cuda_backend, cache.nbytes, zero=False), DeviceBuffer(cuda_backend, pooled.nbytes, zero=False)
    bc.upload(cache)
    bp.upload(pooled)
    q = r.standard_normal((T, H * dk)).astype(np.float32)
    sk = r.standard_normal(H).astype(np.float32)
    op = DeviceOp.cached_attention(0, 1, 2, 2, 3, 0, 0, G * dk, T, H, G, 1, dk, dv, H * dk, width, width, R, dk ** -0.5, mask="pooled", mask_size=size, pooled=4, pool=pool, pool_rows=NB, softcap=cap,
                                   **(dict(sink=5, sink_wdt=abi.W_F32) if shape.get("sink") else {}))
    got = run(cuda_backend, [op], [T * H * dv, q.size, bc.elems, 8 + T, bp.elems, H], [(1, q), (3, ctl_words(pos, 1)), (5, sk)], 0, (T, H, dv), [ExternBuffer(2, bc), ExternBuffer(4, bp)])
    bc.free()
    bp.free()
    p = np.arange(pos, n)[:, None]
    first = max(0, pos + 1 - size)
    j, b = np.arange(first, n), np.arange(NB)
    seen = np.concatenate([(b + 1) * pool <= p + 1 - size, (j <= p) & (j > p - size)], 1)
    rows = np.concatenate([np.nan_to_num(means, nan=0.0), kv[j]]).astype(np.float64)
    want = np.stack([reference(q[:, h * dk:(h + 1) * dk].astype(np.float64), rows[:, h * G // H * dk:(h * G // H + 1) * dk], rows[:, G * dk + h * G // H * dv:G * dk + (h * G // H + 1) * dv], seen,
                               dk ** -0.5, cap, sink=sk[h] if shape.get("sink") else None) for h in range(H)], 1)
    clean = ~sees if bad else np.ones(T, bool)
    assert 0 < clean.sum() and close(got[clean], want[clean])
    assert not bad or not np.isfinite(got[~clean]).any()


def heads_in_a_slab(be, r, T, S, dh, G, H, offs, kv, compile_kv=None):
    """H heads over G slabs of S rows (head h: those that start at row offs[h]) in one buffer, kv[h] keys each -> (got, want, handle, refresh)."""
    from zgml_b200 import DeviceOp, DeviceProgram, ProgramIO
    q, k, v = (r.standard_normal(n).astype(np.float32) for n in ((H, T, dh), (G * S, dh), (G * S, dh)))
    ops = [DeviceOp.attention(3, 0, 1, 2, 0, False, dh, T, (compile_kv or kv)[h], 0.2, h * T * dh, offs[h] * dh, offs[h] * dh, 0, h * T * dh, 1, dh, 1, dh, 1, dh, 0, 0, 1, dh) for h in range(H)]
    handle = be.compile_program(DeviceProgram(ops, [q.size, k.size, v.size, q.size], [], []))
    if compile_kv:
        for o, n in zip(ops, kv):
            o.u.attention.seq_kv = n
        be.refresh_program(handle, ops)
    got = np.zeros((H, T, dh), np.float32)
    be.execute_program(handle, [ProgramIO(i, a.ravel()) for i, a in enumerate((q, k, v))], [ProgramIO(3, got)])
    want = np.empty((H, T, dh))
    for h in range(H):
        kk, vv = (a[offs[h]:offs[h] + kv[h]].astype(np.float64) for a in (k, v))
        want[h] = reference(q[h].astype(np.float64), kk, vv, np.ones((T, kv[h]), bool), 0.2)
    return got, want, handle


def test_scratch_follows_the_slabs(cuda_backend):
    """Eight heads of one buffer: planes for what the operands hold, not for the rest of the buffer behind each head."""
    G, S, dh, T = 8, 640, 64, 40
    got, want, handle = heads_in_a_slab(cuda_backend, np.random.default_rng(13), T, S, dh, G, G, [g * S for g in range(G)], [500] * G)
    assert close(got, want)
    assert 0 < cuda_backend.program_stats(handle)["shared_scratch_elems"] <= 1.1 * 2 * G * S * dh
    cuda_backend.free_program(handle)


def test_more_keys_than_planes(cuda_backend):
    """Head 1 starts at row 128 of head 0's rows when the program is compiled for 100 keys; head 0 is then refreshed past it."""
    got, want, handle = heads_in_a_slab(cuda_backend, np.random.default_rng(14), 70, 400, 64, 1, 2, [0, 128], [390, 150], compile_kv=[100, 100])
    assert close(got, want)
    cuda_backend.free_program(handle)


def test_no_room_for_planes(cuda_backend, monkeypatch):
    monkeypatch.setenv("ZG_CUDA_SCRATCH_MB", "0")
    got, want, handle = heads_in_a_slab(cuda_backend, np.random.default_rng(15), 70, 300, 128, 2, 4, [0, 0, 300, 300], [300, 200, 300, 10])
    assert close(got, want) and cuda_backend.program_stats(handle)["shared_scratch_elems"] == 0
    cuda_backend.free_program(handle)


def test_masks_of_the_lowest_float(cuda_backend):
    """An additive mask that holds the type's lowest value where others hold -inf: beside other scores it weighs nothing; a row that holds nothing else is the
    plain mean of the values (every sum rounds to the lowest value)."""
    from zgml_b200 import DeviceOp, DeviceProgram, ProgramIO
    r = np.random.default_rng(10)
    T, S, dh, H, low = 140, 190, 128, 2, np.finfo(np.float32).min
    q, k, v = r.standard_normal((H, T, dh)).astype(np.float32), r.standard_normal((S, dh)).astype(np.float32), r.standard_normal((S, dh)).astype(np.float32)
    mask = np.where(r.random((T, S)) < 0.5, low, 0.0).astype(np.float32)
    mask[[3, 77, 139]] = low
    ops = [DeviceOp.attention(4, 0, 1, 2, 3, True, dh, T, S, 0.1, h * T * dh, 0, 0, 0, h * T * dh, 1, dh, 1, dh, 1, dh, 1, S, 1, dh) for h in range(H)]
    handle = cuda_backend.compile_program(DeviceProgram(ops, [q.size, k.size, v.size, mask.size, q.size], [], []))
    got = np.zeros((H, T, dh), np.float32)
    cuda_backend.execute_program(handle, [ProgramIO(i, a.ravel()) for i, a in enumerate((q, k, v, mask))], [ProgramIO(4, got)])
    cuda_backend.free_program(handle)
    for h in range(H):
        s = q[h].astype(np.float64) @ k.astype(np.float64).T * 0.1 + mask
        s[[3, 77, 139]] = 0.0
        e = np.exp(s - s.max(1, keepdims=True))
        assert close(got[h], e @ v.astype(np.float64) / e.sum(1, keepdims=True))


@pytest.mark.parametrize("what", ["nan key", "nan value", "infinite value"])
def test_batched_rows_that_see_nothing_non_finite_are_exact(cuda_backend, what):
    """DeviceOp.attention: position 70 of the first of two key / value slabs holds no number; the rows whose mask leaves it out, and the heads of the other
    slab, are as they were."""
    from zgml_b200 import DeviceOp, DeviceProgram, ProgramIO
    r = np.random.default_rng(9)
    T, S, dh, H = 150, 200, 64, 4
    q, k, v = r.standard_normal((H, T, dh)).astype(np.float32), r.standard_normal((2, S, dh)).astype(np.float32), r.standard_normal((2, S, dh)).astype(np.float32)
    (k if what == "nan key" else v)[0, 70] = np.inf if what == "infinite value" else np.nan
    mask = np.where(r.random((T, S)) < 0.5, -np.inf, 0.0).astype(np.float32)
    ops = [DeviceOp.attention(4, 0, 1, 2, 3, True, dh, T, S, 0.3, h * T * dh, h % 2 * S * dh, h % 2 * S * dh, 0, h * T * dh, 1, dh, 1, dh, 1, dh, 1, S, 1, dh) for h in range(H)]
    handle = cuda_backend.compile_program(DeviceProgram(ops, [q.size, k.size, v.size, mask.size, q.size], [], []))
    got = np.zeros((H, T, dh), np.float32)
    cuda_backend.execute_program(handle, [ProgramIO(i, a.ravel()) for i, a in enumerate((q, k, v, mask))], [ProgramIO(4, got)])
    cuda_backend.free_program(handle)
    sees = mask[:, 70] == 0.0
    for h in range(H):
        rows = ~sees if h % 2 == 0 else np.ones(T, bool)
        kk, vv = np.where(np.isfinite(k[h % 2]), k[h % 2], 0.0).astype(np.float64), np.where(np.isfinite(v[h % 2]), v[h % 2], 0.0).astype(np.float64)
        s = q[h].astype(np.float64) @ kk.T * 0.3 + mask
        e = np.exp(s - s.max(1, keepdims=True))
        want = e @ vv / e.sum(1, keepdims=True)
        assert close(got[h][rows], want[rows])
        # a NaN score counts as masked there, a value that is no number does not
        assert what == "nan key" or h % 2 or not np.isfinite(got[h][sees]).any()


def test_no_wait_ran_out(cuda_backend):
    """After everything above: a wait that gives up is counted (and its rows are no numbers)."""
    assert waits_given_up(cuda_backend) == 0
