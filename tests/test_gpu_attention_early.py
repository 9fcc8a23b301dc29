"""CACHED_ATTENTION of few rows reads the cache's rows of earlier positions before its predecessor has completed where all that the program writes into the cache are
the step's own rows: positions around the 32 of a buffer and a share's edges, rings that are just large enough, several steps in a row — against the same program without a
graph, where nothing is read ahead.  And programs in which something else writes a row that the step sees, right before it: the rule must leave those alone."""
import numpy as np
import pytest

from test_gpu_recops import ctl_words

pytestmark = pytest.mark.gpu


def program(be, T, H, G, dk, dv, R, mask="causal", size=0, patch=None):
    """append -> attention over one cache [R, G (dk + dv)]; patch: a second append in between, at the position of its own control words (or of the step's, "narrow": one token)"""
    from zgml_b200 import DeviceBuffer, DeviceOp, DeviceProgram, ExternBuffer
    width = G * (dk + dv)
    rs = H * dk + width
    kept = DeviceBuffer(be, 4 * R * width)
    sizes = [T * H * dv, T * rs, 8 + T, R * width, 8 + T, T * rs]
    ops = [DeviceOp.cache_append(3, 1, 2, H * dk, 0, T, width, rs, width, R)]
    if patch:
        ops.append(DeviceOp.cache_append(3, 5, 4, H * dk, 0, 1 if patch == "narrow" else T, width, rs, width, R))
    ops.append(DeviceOp.cached_attention(0, 1, 3, 3, 2, 0, 0, G * dk, T, H, G, 1, dk, dv, rs, width, width, R, dk ** -0.5, mask=mask, mask_size=size))
    h = be.compile_program(DeviceProgram(ops, sizes, [], [], [ExternBuffer(3, kept)]))
    assert h is not None
    return h, kept, width, rs


def step(be, h, T, H, dv, pos, x, pos2=0, y=None):
    from zgml_b200 import ProgramIO
    got = np.zeros((T, H, dv), np.float32)
    io = [ProgramIO(1, x.ravel()), ProgramIO(2, ctl_words(pos, 0, 8 + T))]
    if y is not None:
        io += [ProgramIO(4, ctl_words(pos2, 0, 8 + T)), ProgramIO(5, y.ravel())]
    be.execute_program(h, io, [ProgramIO(0, got)])
    return got


@pytest.mark.parametrize("T,H,G,dk,dv,R,mask,size", [(1, 16, 1, 576, 512, 400, "causal", 0), (1, 8, 2, 64, 64, 700, "causal", 0), (3, 4, 1, 128, 96, 300, "causal", 0),
                                                     (2, 4, 2, 36, 64, 65, "window", 64), (1, 4, 4, 64, 32, 33, "window", 33)])
def test_read_ahead_as_without(cuda_backend, T, H, G, dk, dv, R, mask, size):
    r = np.random.default_rng(T + dk)
    h, kept, width, rs = program(cuda_backend, T, H, G, dk, dv, R, mask, size)
    got = {True: [], False: []}
    rows = r.standard_normal((R, width)).astype(np.float32)
    at = [p for p in (0, 1, 30, 31, 32, 33, 62, 63, 64, 65, 127, 300) if mask == "window" or p + T <= R]
    xs = [r.standard_normal((T, rs)).astype(np.float32) for _ in at]
    try:
        for graph in (True, False):
            cuda_backend.set_graph_mode(graph)
            kept.upload(rows)
            for p, x in zip(at, xs):
                got[graph].append(step(cuda_backend, h, T, H, dv, p, x))
    finally:
        cuda_backend.set_graph_mode(True)
    for p, a, b in zip(at, got[True], got[False]):
        assert np.array_equal(a, b), p
    cuda_backend.free_program(h)
    kept.free()


@pytest.mark.parametrize("patch,pos2", [("other", 40), ("other", 3), ("narrow", 7)])
def test_rows_that_something_else_writes_are_waited_for(cuda_backend, patch, pos2):
    T, H, G, dk, dv, R, pos = 2, 4, 1, 64, 64, 64, 50
    r = np.random.default_rng(pos2)
    h, kept, width, rs = program(cuda_backend, T, H, G, dk, dv, R, patch=patch)
    for _ in range(5):
        rows = r.standard_normal((R, width)).astype(np.float32)
        kept.upload(rows)
        x, y = (r.standard_normal((T, rs)).astype(np.float32) for _ in range(2))
        got = step(cuda_backend, h, T, H, dv, pos, x, pos2, y)
        n = 1 if patch == "narrow" else T
        rows[pos:pos + T] = x[:, H * dk:]
        rows[pos2:pos2 + n] = y[:n, H * dk:]
        k, v = rows[:, :dk].astype(np.float64), rows[:, dk:].astype(np.float64)
        for t in range(T):
            s = x[t, :H * dk].reshape(H, dk).astype(np.float64) @ k[:pos + t + 1].T * dk ** -0.5
            e = np.exp(s - s.max(-1, keepdims=True))
            want = e / e.sum(-1, keepdims=True) @ v[:pos + t + 1]
            assert np.abs(got[t] - want).max() <= 1e-5 * np.abs(want).max()      # 24-bit operands, f32 sums of 50 terms
    cuda_backend.free_program(h)
    kept.free()
