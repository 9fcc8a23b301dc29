"""LINEAR of many rows over f32 weights where the source is cut ahead (four and more 64-k steps a CTA) against float64: K on and off the planes' eight
elements, a last step of four elements, rows and weight rows on and off the tiles, several shares of K, a source that is a slot of a state buffer of which
only some rows count, and elements that are not finite.  Bounds as in test_gpu_split_gemm.py."""
import numpy as np
import pytest

from test_gpu_recops import ctl_words, run, weights
from test_gpu_split_gemm import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(9, 2500, 256), (128, 257, 260), (129, 128, 324), (40, 20000, 388), (257, 130, 1028), (10, 33, 4100)])
def test_source_cut_ahead(cuda_backend, M, N, K):
    from zgml_b200 import DeviceOp, ExternBuffer, abi
    r = np.random.default_rng(M + N + K)
    W = (r.standard_normal((N, K)) * 10.0 ** r.integers(-12, 12, (N, 1))).astype(np.float32)
    x = (r.standard_normal((M, K)) * 10.0 ** r.integers(-9, 9, (M, 1))).astype(np.float32)
    buf, (ow,) = weights(cuda_backend, W)
    op = DeviceOp.linear(0, 1, 2, ow, M, N, K, abi.W_F32)
    got = run(cuda_backend, [op], [M * N, x.size, buf.elems], [(1, x)], 0, (M, N), [ExternBuffer(2, buf)])
    check(got, x, W, x.astype(np.float64) @ W.astype(np.float64).T)
    buf.free()


def test_non_finite_elements(cuda_backend):
    from zgml_b200 import DeviceOp, ExternBuffer, abi
    r = np.random.default_rng(2)
    M, N, K = 40, 64, 640
    W, x = r.standard_normal((N, K)).astype(np.float32), r.standard_normal((M, K)).astype(np.float32)
    x[3, 70], x[17, 5], W[9, 9] = np.inf, np.nan, -np.inf
    buf, (ow,) = weights(cuda_backend, W)
    got = run(cuda_backend, [DeviceOp.linear(0, 1, 2, ow, M, N, K, abi.W_F32)], [M * N, x.size, buf.elems], [(1, x)], 0, (M, N), [ExternBuffer(2, buf)])
    with np.errstate(invalid="ignore"):
        want = x.astype(np.float64) @ W.astype(np.float64).T
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))
    rows, cols = np.delete(np.arange(M), [3, 17]), np.delete(np.arange(N), 9)
    check(got[np.ix_(rows, cols)], x[rows], W[cols], want[np.ix_(rows, cols)])
    buf.free()


def test_rows_of_a_slot(cuda_backend):
    from zgml_b200 import DeviceBuffer, DeviceOp, ExternBuffer, abi
    r = np.random.default_rng(4)
    M, N, K, slot, pos, live = 300, 70, 516, 2, 100, 40       # rows below 140 count
    W, state = r.standard_normal((N, K)).astype(np.float32), r.standard_normal((3, M, K)).astype(np.float32)
    buf, (ow,) = weights(cuda_backend, W)
    st = DeviceBuffer(cuda_backend, 4 * state.size)
    st.upload(state.ravel())
    op = DeviceOp.linear(0, 1, 2, ow, M, N, K, abi.W_F32, ctl=3, src_slot_stride=M * K, live_rows=live)
    got = run(cuda_backend, [op], [M * N, st.elems, buf.elems, 8], [(3, ctl_words(pos, slot))], 0, (M, N), [ExternBuffer(2, buf), ExternBuffer(1, st)])
    n = pos + live
    check(got[:n], state[slot, :n], W, state[slot, :n].astype(np.float64) @ W.astype(np.float64).T)
    buf.free()
    st.free()
