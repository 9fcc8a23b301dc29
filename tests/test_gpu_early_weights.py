"""NORM of few rows and STREAM_STEP read weights before their predecessor has completed only where nothing in the program writes them.  Here the op before copies the
weight into its place: the same program, executed with one weight after the other, would answer with the one of the pass before.

Tolerance: as in the widths' tests (1e-5 of the largest output for a norm of f32 sums)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def copy(to, frm, n):
    from zgml_b200 import DeviceOp
    return DeviceOp.slice_assign(to, frm, n, 1, 0, 0, 1, n, 0, 1, n, 0)


def passes(be, ops, sizes, inputs, weight_src, weight, want, outs):
    """Executes the program with six weights; want(weight) -> {buffer: array}."""
    from zgml_b200 import DeviceProgram, ProgramIO
    h = be.compile_program(DeviceProgram(ops, sizes))
    assert be.program_stats(h)["early_weight_norms"] == 0
    for seed in range(6):
        w = weight(np.random.default_rng(seed))
        got = {b: np.zeros(s, np.float32) for b, s in outs.items()}
        be.execute_program(h, [ProgramIO(i, a.ravel()) for i, a in inputs] + [ProgramIO(weight_src, w.ravel())], [ProgramIO(b, g) for b, g in got.items()])
        for b, v in want(w.astype(np.float64)).items():
            assert np.abs(got[b] - v).max() <= 1e-5 * max(1.0, np.abs(v).max()), (seed, b)
    be.free_program(h)


def rms(v):
    v = v.astype(np.float64)
    return v / np.sqrt((v ** 2).mean(-1, keepdims=True) + 1e-5)


@pytest.mark.parametrize("rows", [1, 8, 63])
@pytest.mark.parametrize("form", ["alone", "chained", "residual", "dyt"])
def test_norm(cuda_backend, form, rows):
    from zgml_b200 import DeviceOp, abi
    cols = 1500
    r = np.random.default_rng(rows)
    x, res, fixed = r.standard_normal((rows, cols)).astype(np.float32), r.standard_normal((rows, cols)).astype(np.float32), r.standard_normal(cols).astype(np.float32)
    n = 2 * cols + 1 if form == "dyt" else cols
    # 0 out, 1 x, 2 written weight, 3 residual, 4 chained out, 5 where the weight comes from, 6 a weight that nothing writes
    sizes, inputs = [x.size, x.size, n, x.size, x.size, n, cols], [(1, x), (3, res), (6, fixed)]
    if form == "alone":
        op, want = DeviceOp.norm(0, 1, 2, 0, rows, cols, 1e-5, abi.W_F32, kind="rms"), lambda w: {0: rms(x) * w}
    elif form == "chained":
        op = DeviceOp.norm(0, 1, 6, 0, rows, cols, 1e-5, abi.W_F32, kind="rms", then=4, then_w=2, then_kind="rms")
        want = lambda w: {0: rms(x) * fixed, 4: rms(rms(x) * fixed) * w}
    elif form == "residual":
        op = DeviceOp.norm(0, 1, 2, 0, rows, cols, 1e-5, abi.W_F32, kind="none", res=3, then=4, then_w=2, then_kind="rms")
        want = lambda w: {0: res.astype(np.float64) + x, 4: rms(res.astype(np.float64) + x) * w}
    else:
        op = DeviceOp.norm(0, 1, 2, 0, rows, cols, 1e-5, abi.W_F32, kind="dyt", res=3)
        want = lambda w: {0: res + np.tanh(w[2 * cols] * x) * w[:cols] + w[cols:2 * cols]}
    outs = {0: x.shape} if form in ("alone", "dyt") else {0: x.shape, 4: x.shape}
    passes(cuda_backend, [copy(2, 5, n), op], sizes, inputs, 5, lambda g: g.standard_normal(n).astype(np.float32), want, outs)


@pytest.mark.parametrize("T", [1, 9])
@pytest.mark.parametrize("side", ["close", "open"])
def test_stream_step(cuda_backend, side, T):
    from zgml_b200 import DeviceOp, abi
    S, D = 2, 600
    r = np.random.default_rng(T)
    X, y = r.standard_normal((S, T, D)).astype(np.float32), r.standard_normal((T, D)).astype(np.float32)
    n = S + S * S + D if side == "close" else S + 2 * D + 1
    # 0 new streams, 1 streams, 2 y, 3 written weights, 4 opened input, 5 where they come from
    sizes, inputs = [X.size, X.size, y.size, n, y.size, n], [(1, X), (2, y)]
    if side == "close":
        op = DeviceOp.stream_step(T, D, S, abi.W_F32, dst=0, src=1, src_stride=T * D, y=2, close_w=3, out_off=0, mix_off=S, ls_off=S + S * S, mult=0.7)
        want = lambda w: {0: np.einsum("ab,atd->btd", w[S:S + S * S].reshape(S, S), X) + 0.7 * w[:S, None, None] * (y * w[S + S * S:])[None]}
        outs = {0: X.shape}
    else:
        op = DeviceOp.stream_step(T, D, S, abi.W_F32, src=1, src_stride=T * D, h=4, open_w=3, in_off=0, norm_off=S)
        want = lambda w: {4: np.tanh(w[S + 2 * D] * np.tensordot(w[:S], X.astype(np.float64), (0, 0))) * w[S:S + D] + w[S + D:S + 2 * D]}
        outs = {4: y.shape}
    passes(cuda_backend, [copy(3, 5, n), op], sizes, inputs, 5, lambda g: g.standard_normal(n).astype(np.float32), want, outs)


def test_weights_that_nothing_writes_are_read_ahead(cuda_backend):
    from zgml_b200 import DeviceOp, DeviceProgram, abi
    op = DeviceOp.norm(0, 1, 2, 0, 1, 64, 1e-5, abi.W_F32, kind="rms", then=3, then_w=4, then_kind="rms")
    for ops, early in (([op], 1), ([copy(2, 5, 64), op], 0), ([copy(4, 5, 64), op], 0)):
        h = cuda_backend.compile_program(DeviceProgram(ops, [64] * 6))
        assert cuda_backend.program_stats(h)["early_weight_norms"] == early
        cuda_backend.free_program(h)
