"""Sequence ops where the scratch that their faster forms stage in cannot be had (ZG_CUDA_SCRATCH_MB refuses every allocation): the program compiles all the same
and the forms without scratch answer as the others do.

Where only the LINEAR's cut source has no room, the form that cuts it as it goes gives the same sums, bit for bit.

Tolerance: two f32 evaluations of the same sums, each within 1e-5 of the result's largest value of the true one (the bars of the ops' own tests)."""
import numpy as np
import pytest

from test_gpu_recops import ctl_words, run, weights

pytestmark = pytest.mark.gpu


def linear(be, r):
    from zgml_b200 import DeviceOp, ExternBuffer, abi
    M, N, K = 40, 70, 4096
    w, (ow,) = weights(be, r.standard_normal((N, K)))
    x = r.standard_normal((M, K)).astype(np.float32)
    return [DeviceOp.linear(0, 1, 2, ow, M, N, K, abi.W_F32)], [M * N, x.size, w.elems], [(1, x)], (M, N), [ExternBuffer(2, w)], [w]


def attention(be, r, T=200):
    from zgml_b200 import DeviceBuffer, DeviceOp, ExternBuffer
    pos, H, d = 200, 8, 128
    rows = r.standard_normal((pos + T, H * d)).astype(np.float32)
    cache = DeviceBuffer(be, rows.nbytes, zero=False)
    cache.upload(rows)
    q = r.standard_normal((T, H * d)).astype(np.float32)
    op = DeviceOp.cached_attention(0, 1, 2, 2, 3, 0, 0, 0, T, H, H, 1, d, d, H * d, H * d, H * d, pos + T, d ** -0.5, mask="causal")
    return [op], [T * H * d, q.size, cache.elems, 8 + T], [(1, q), (3, ctl_words(pos, 0))], (T, H, d), [ExternBuffer(2, cache)], [cache]


def one_token(be, r):
    return attention(be, r, 1)


def delta_rule(be, r):
    from zgml_b200 import DeviceBuffer, DeviceOp, ExternBuffer, abi
    T, H, dim, vdim = 50, 2, 64, 32
    w, (oA, odt, onw) = weights(be, r.standard_normal(H), r.standard_normal((H, dim)), 1 + 0.2 * r.standard_normal(vdim))
    qrs = 2 * H * dim + 2 * H * vdim + H
    proj, a = r.standard_normal((T, qrs)).astype(np.float32), r.standard_normal((T, H * dim)).astype(np.float32)
    state = DeviceBuffer(be, 4 * H * dim * vdim)
    op = DeviceOp.delta_rule(0, 1, 1, 2, 1, 3, 4, 5, 0, H * dim, 2 * H * dim, 2 * H * dim + 2 * H * vdim, oA, odt, onw, T, H, H, dim, vdim, qrs, qrs, H * dim, qrs, abi.W_F32, 1e-5, 1e-6, 0.4,
                             gate_off=2 * H * dim + H * vdim)
    return [op], [T * H * vdim, proj.size, a.size, w.elems, state.elems, 8], [(1, proj), (2, a), (5, ctl_words(0, 0))], (T, H, vdim), [ExternBuffer(3, w), ExternBuffer(4, state)], [w, state]


def ssm_scan(be, r):
    from zgml_b200 import DeviceBuffer, DeviceOp, ExternBuffer, abi
    from zgml_b200.backend import seq_state_elems
    T, H, N, P = 200, 2, 64, 64
    xbc, dt = r.standard_normal((T, H * P + 2 * N)).astype(np.float32), r.standard_normal((T, H)).astype(np.float32)
    w, offs = weights(be, r.standard_normal(H), r.standard_normal(H), r.standard_normal(H))
    args = (0, H * P, H * P + N, 0, *offs, T, H, 1, N, P, xbc.shape[1], H, abi.W_F32)
    state = DeviceBuffer(be, 4 * seq_state_elems(DeviceOp.ssm_scan(0, 1, 2, 3, 4, 5, *args)))
    return [DeviceOp.ssm_scan(0, 1, 2, 3, 4, 5, *args)], [T * H * P, xbc.size, dt.size, w.elems, state.elems, 8], [(1, xbc), (2, dt), (5, ctl_words(0, 0))], (T, H, P), \
        [ExternBuffer(3, w), ExternBuffer(4, state)], [w, state]


@pytest.mark.parametrize("make", [linear, attention, one_token, delta_rule, ssm_scan])
def test_without_scratch(cuda_backend, monkeypatch, make):
    outs = []
    for limit in (None, "0"):
        if limit:
            monkeypatch.setenv("ZG_CUDA_SCRATCH_MB", limit)
        ops, sizes, io, shape, ext, owned = make(cuda_backend, np.random.default_rng(20))
        outs.append(run(cuda_backend, ops, sizes, io, 0, shape, ext))
        for b in owned:
            b.free()
    assert np.abs(outs[0] - outs[1]).max() <= 2e-5 * np.abs(outs[0]).max()


def test_without_room_for_the_cut_source(cuda_backend, monkeypatch):
    """150 tiles of one share each: the parts of the source are all that it stages (1.8 MB)."""
    from zgml_b200 import DeviceOp, ExternBuffer, abi
    r = np.random.default_rng(3)
    M, N, K = 600, 3800, 512
    w, (ow,) = weights(cuda_backend, r.standard_normal((N, K)))
    x = r.standard_normal((M, K)).astype(np.float32)
    outs = []
    for limit in (None, "1"):
        if limit:
            monkeypatch.setenv("ZG_CUDA_SCRATCH_MB", limit)
        outs.append(run(cuda_backend, [DeviceOp.linear(0, 1, 2, ow, M, N, K, abi.W_F32)], [M * N, x.size, w.elems], [(1, x)], 0, (M, N), [ExternBuffer(2, w)]))
    assert np.array_equal(outs[0], outs[1])
    w.free()
