"""NORM of few rows at the widths where the threads per row change: the step that closes a sublayer and opens the next (dst = res + src, then = rms(dst) w), and
two sources, each normed on its own (dst = res + outer(rms(src) w + rms(src2) w2), then = rms(dst) w3).

Tolerance: a sum of 4097 squares in f32, four to a thread and then over lanes and warps, is off by less than 2^-20 of itself, its root by half of that: 1e-5 of the
largest output leaves room for the division and two products.  With two sources two or three such norms follow one another: 2e-5."""
import numpy as np
import pytest

from test_gpu_recops import run, weights

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


@pytest.mark.parametrize("cols", [1024, 1025, 2048, 2049, 3000, 4095, 4096, 4097])
@pytest.mark.parametrize("outer", [False, True], ids=["plain", "outer"])
@pytest.mark.parametrize("kind", ["rms", "layer"])
def test_two_sources(cuda_backend, kind, outer, cols):
    """The sources' sizes differ by 30, so that sums that were mixed up would show."""
    from zgml_b200 import DeviceOp, ExternBuffer, abi
    r = np.random.default_rng(cols)
    rows = 2
    x, y, res = (s * r.standard_normal((rows, cols)).astype(np.float32) for s in (np.float32(1), np.float32(30), np.float32(1)))
    w = (1 + 0.3 * r.standard_normal((4, cols))).astype(np.float32)
    buf, offs = weights(cuda_backend, *w)
    op = DeviceOp.norm(0, 1, 2, offs[0], rows, cols, 1e-5, abi.W_F32, kind=kind, res=3, src2=5, src2_w_off=offs[1], outer=kind if outer else None, outer_w_off=offs[2], then=4, then_w=2,
                       then_w_off=offs[3], then_kind="rms")

    def normed(v, i, mean=kind == "layer"):
        v = v - v.mean(1, keepdims=True) if mean else v
        return v / np.sqrt((v ** 2).mean(1, keepdims=True) + 1e-5) * w[i].astype(np.float64)
    total = normed(x.astype(np.float64), 0) + normed(y.astype(np.float64), 1)
    total = res + (normed(total, 2) if outer else total)
    sizes, io = [x.size, x.size, buf.elems, x.size, x.size, x.size], [(1, x), (3, res), (5, y)]
    for out, want in ((0, total), (4, normed(total, 3, False))):
        got = run(cuda_backend, [op], sizes, io, out, x.shape, [ExternBuffer(2, buf)])
        assert np.abs(got - want).max() <= 2e-5 * np.abs(want).max()
    buf.free()


@pytest.mark.parametrize("cols", [512, 513, 1024, 1025, 2048, 2049, 4096, 4097])
@pytest.mark.parametrize("more", [0, 1], ids=["one-wave", "past-it"])
def test_many_rows(cuda_backend, cols, more):
    """The largest count of rows that is resident at once, and one row more.  The weight comes from a launch of the same program."""
    import torch
    from zgml_b200 import DeviceOp, abi
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows = sms * (4 if cols <= 1024 else 2 if cols <= 2048 else 1) + more
    r = np.random.default_rng(cols)
    x, res = (r.standard_normal((rows, cols)).astype(np.float32) for _ in range(2))
    w, ones = (1 + 0.3 * r.standard_normal((1, cols))).astype(np.float32), np.ones((2 * cols,), np.float32)
    ops = [DeviceOp.norm(2, 5, 6, 0, 1, cols, 1e-5, abi.W_F32, kind="rms"), DeviceOp.norm(0, 1, 2, 0, rows, cols, 1e-5, abi.W_F32, kind="none", res=3, then=4, then_w=2, then_w_off=0, then_kind="rms")]
    sizes, io = [x.size, x.size, cols, x.size, x.size, cols, ones.size], [(1, x), (3, res), (5, w), (6, ones)]
    wn = w / np.sqrt((w.astype(np.float64) ** 2).mean() + 1e-5)
    total = res.astype(np.float64) + x
    for out, want in ((0, total), (4, total / np.sqrt((total ** 2).mean(1, keepdims=True) + 1e-5) * wn)):
        got = run(cuda_backend, ops, sizes, io, out, x.shape)
        assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
