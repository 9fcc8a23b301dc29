"""NORM of few rows that closes a sublayer and opens the next (dst = res + src, then = rms(dst) w) at the widths where the threads per row change.

Tolerance: a sum of 4097 squares in f32, four to a thread and then over lanes and warps, is off by less than 2^-20 of itself, its root by half of that: 1e-5 of the
largest output leaves room for the division and two products."""
import numpy as np
import pytest

from test_gpu_recops import run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [1, 255, 1024, 1025, 2047, 2048, 2049, 3000, 4096, 4097])
@pytest.mark.parametrize("rows", [1, 3])
def test_residual_then_rms(cuda_backend, rows, cols):
    from zgml_b200 import DeviceBuffer, DeviceOp, ExternBuffer, abi
    r = np.random.default_rng(cols + rows)
    x, res, w = (r.standard_normal(s).astype(np.float32) for s in ((rows, cols), (rows, cols), (cols,)))
    buf = DeviceBuffer(cuda_backend, w.nbytes, zero=False)
    buf.upload(w)
    op = DeviceOp.norm(0, 1, 2, 0, rows, cols, 1e-5, abi.W_F32, kind="none", res=3, then=4, then_w=2, then_w_off=0, then_kind="rms")
    sizes, io = [x.size, x.size, buf.elems, x.size, x.size], [(1, x), (3, res)]
    total = res.astype(np.float64) + x
    for out, want in ((0, total), (4, total / np.sqrt((total ** 2).mean(1, keepdims=True) + 1e-5) * w)):
        got = run(cuda_backend, [op], sizes, io, out, x.shape, [ExternBuffer(2, buf)])
        assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
    buf.free()
