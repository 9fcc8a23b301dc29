"""Two threads with a backend each compile and run programs whose launches of one kernel ask for different amounts of shared memory: the limit that either sets is
enough for the other's launch, whatever the order."""
import threading

import numpy as np
import pytest

from test_gpu_recops import ctl_words, run, weights

pytestmark = pytest.mark.gpu


def linear(be, large):
    from zgml_b200 import DeviceOp, ExternBuffer, abi
    N, K = (64, 16384) if large else (3100, 512)
    r = np.random.default_rng(K)
    w, (ow,) = weights(be, r.standard_normal((N, K)))
    return [DeviceOp.linear(0, 1, 2, ow, 1, N, K, abi.W_F32)], [N, K, w.elems], [(1, r.standard_normal(K))], (N,), [ExternBuffer(2, w)], [w]


def delta_rule(be, large):
    from zgml_b200 import DeviceBuffer, DeviceOp, ExternBuffer, abi
    T, H, dim, vdim = 64, 2 if large else 160, 64, 16      # three stages, two
    r = np.random.default_rng(H)
    w, (oA, odt, onw) = weights(be, r.standard_normal(H), r.standard_normal((H, dim)), 1 + 0.2 * r.standard_normal(vdim))
    qrs = 2 * H * dim + 2 * H * vdim + H
    proj, a = r.standard_normal((T, qrs)), r.standard_normal((T, H * dim))
    state = DeviceBuffer(be, 4 * H * dim * vdim)
    op = DeviceOp.delta_rule(0, 1, 1, 2, 1, 3, 4, 5, 0, H * dim, 2 * H * dim, 2 * H * dim + 2 * H * vdim, oA, odt, onw, T, H, H, dim, vdim, qrs, qrs, H * dim, qrs, abi.W_F32, 1e-5, 1e-6, 0.4,
                             gate_off=2 * H * dim + H * vdim)
    return [op], [T * H * vdim, proj.size, a.size, w.elems, state.elems, 8], [(1, proj), (2, a), (5, ctl_words(0, 0))], (T, H, vdim), [ExternBuffer(3, w), ExternBuffer(4, state)], [w, state]


def attention(be, large):
    from zgml_b200 import DeviceBuffer, DeviceOp, ExternBuffer
    H, d, dv, R = 4, 512 if large else 64, 64, 512
    r = np.random.default_rng(d)
    k, v = DeviceBuffer(be, 4 * R * d, zero=False), DeviceBuffer(be, 4 * R * dv, zero=False)
    k.upload(r.standard_normal(R * d).astype(np.float32))
    v.upload(r.standard_normal(R * dv).astype(np.float32))
    op = DeviceOp.cached_attention(0, 1, 2, 3, 4, 0, 0, 0, 1, H, 1, 1, d, dv, H * d, d, dv, R, d ** -0.5, mask="causal")
    return [op], [H * dv, H * d, k.elems, v.elems, 8], [(1, r.standard_normal(H * d)), (4, ctl_words(R - 1, 0))], (H, dv), [ExternBuffer(2, k), ExternBuffer(3, v)], [k, v]


@pytest.mark.parametrize("make", [linear, delta_rule, attention])
def test_two_threads(make):
    from zgml_b200 import CudaBackend
    failed = []

    def work(large):
        try:
            be = CudaBackend(0)
            ops, sizes, io, shape, ext, owned = make(be, large)
            state = owned[-1].download(np.float32, 0, owned[-1].elems)
            first = None
            for _ in range(200):
                owned[-1].upload(state)                    # (the delta rule's changes from run to run)
                got = run(be, ops, sizes, io, 0, shape, ext)
                first = got if first is None else first
                assert np.isfinite(got).all() and np.array_equal(got, first)
            for b in owned:
                b.free()
            be.close()
        except BaseException as e:  # noqa: BLE001
            failed.append((large, e))
    threads = [threading.Thread(target=work, args=(large,)) for large in (False, True)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
