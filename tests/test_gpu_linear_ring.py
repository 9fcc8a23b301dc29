"""LINEAR of up to eight rows over enough weight for the ring of slots: K within one piece of a row, of several and with a short last one, where 32, 64, 128 and
256 threads share a row, fewer outputs than SMs and counts that do not divide among them, pairs just below and above what asks for the ring, activations that fit
shared memory and those that pass through in segments of K, strided and unaligned rows, rows of a state buffer's slot, and a weight that the program itself writes.

Tolerance: a sum is added up in chains of at most 16 elements per 4 KB piece of a row (64 for K = 16384), then over 256 threads in a tree: below 100 roundings
of 2^-24 of the sum of magnitudes."""
import numpy as np
import pytest

from test_gpu_recops import ctl_words, run

pytestmark = pytest.mark.gpu


def _bf16(a):
    u = np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)
    return ((u + np.uint32(0x7FFF) + ((u >> np.uint32(16)) & np.uint32(1))) & np.uint32(0xFFFF0000)).view(np.float32)


def _silu(z):
    return z / (1.0 + np.exp(-z))


@pytest.mark.parametrize("M,N,K,fmt", [(1, 3100, 256, "bfloat16"), (1, 1600, 520, "bfloat16"), (2, 149, 2056, "float32"), (1, 147, 8200, "bfloat16"), (3, 1033, 1000, "bfloat16"),
                                       (4, 777, 512, "float32"), (5, 301, 4104, "bfloat16"), (8, 297, 6144, "bfloat16"), (8, 150, 3076, "float32"), (2, 64, 16384, "bfloat16"),
                                       (7, 40, 12296, "bfloat16"), (1, 60000, 32, "bfloat16"), (1, 1024, 568, "bfloat16"), (1, 1024, 576, "bfloat16"), (4, 1024, 144, "float32")])
@pytest.mark.parametrize("pairs", [False, True], ids=["rows", "pairs"])
def test_linear_rows_through_the_ring(cuda_backend, M, N, K, fmt, pairs):
    from zgml_b200 import DeviceOp, ExternBuffer, abi
    from zgml_b200.host.weights import WeightArena
    wdt = abi.W_F32 if fmt == "float32" else abi.W_BF16
    r = np.random.default_rng(N + K)
    W, b = _bf16(r.standard_normal((N * (2 if pairs else 1), K)) / np.sqrt(K)), _bf16(0.3 * r.standard_normal(N))
    A = WeightArena(wdt)
    ow, ob = A.add("w", W), A.add("b", b)
    buf = A.upload(cuda_backend)
    srs, drs = K + 4, N + 3
    x = r.standard_normal((M, srs)).astype(np.float32)
    xx, ww = x[:, :K].astype(np.float64), W.astype(np.float64)
    z, mag = xx @ ww.T, np.abs(xx) @ np.abs(ww).T
    for unaligned in (0, 1):                               # activations at a 16-byte boundary or not
        src = np.zeros(unaligned + x.size, np.float32)
        src[unaligned:] = x.ravel()
        if pairs:
            op = DeviceOp.linear(0, 1, 2, ow, M, N, K, wdt, act="silu", pairs=True, src_off=unaligned, src_rs=srs, dst_rs=drs)
            g, u = z[:, 0::2], z[:, 1::2]
            want, room = _silu(g) * u, 100 * 2.0 ** -24 * (1.2 * mag[:, 0::2] * np.abs(u) + mag[:, 1::2] * np.abs(_silu(g)) + 1e-2)
        else:
            op = DeviceOp.linear(0, 1, 2, ow, M, N, K, wdt, bias=2, bias_off=ob, src_off=unaligned, src_rs=srs, dst_rs=drs)
            want, room = z + b, 100 * 2.0 ** -24 * (mag + np.abs(b))
        got = run(cuda_backend, [op], [M * drs, src.size, buf.elems], [(1, src)], 0, (M, drs), [ExternBuffer(2, buf)])[:, :N]
        assert (np.abs(got - want) <= room).all(), unaligned
    buf.free()


@pytest.mark.parametrize("M,K", [(1, 2056), (2, 2056), (3, 1032), (4, 4104), (8, 1032), (8, 6144)])
@pytest.mark.parametrize("extra", [0, 1, 2, 3])
@pytest.mark.parametrize("fmt", ["bfloat16", "float32"])
def test_rows_of_a_slot(cuda_backend, fmt, extra, M, K):
    """The source is the second slot of a state buffer whose slots lie any number of elements apart."""
    from zgml_b200 import DeviceBuffer, DeviceOp, ExternBuffer, abi
    from zgml_b200.host.weights import WeightArena
    wdt = abi.W_F32 if fmt == "float32" else abi.W_BF16
    r = np.random.default_rng(K + extra)
    N, stride = 777, M * K + extra
    W = _bf16(r.standard_normal((N, K)) / np.sqrt(K))
    A = WeightArena(wdt)
    ow = A.add("w", W)
    buf = A.upload(cuda_backend)
    slots = r.standard_normal(2 * stride).astype(np.float32)
    state = DeviceBuffer(cuda_backend, slots.nbytes, zero=False)
    state.upload(slots)
    x, ww = slots[stride:stride + M * K].reshape(M, K).astype(np.float64), W.astype(np.float64)
    op = DeviceOp.linear(0, 1, 2, ow, M, N, K, wdt, ctl=3, src_slot_stride=stride)
    got = run(cuda_backend, [op], [M * N, state.elems, buf.elems, 8], [(3, ctl_words(0, 1))], 0, (M, N), [ExternBuffer(2, buf), ExternBuffer(1, state)])
    assert (np.abs(got - x @ ww.T) <= 100 * 2.0 ** -24 * (np.abs(x) @ np.abs(ww).T)).all()
    buf.free()
    state.free()


def test_a_weight_that_the_program_writes_is_read_after_it(cuda_backend):
    """The weight is copied into its place by the op before: the same program, executed with one weight after the other, would answer with the one of the pass before."""
    from zgml_b200 import DeviceOp, DeviceProgram, ProgramIO, abi
    r = np.random.default_rng(3)
    N, K = 2048, 2048
    x = r.standard_normal(K).astype(np.float32)
    ops = [DeviceOp.slice_assign(2, 3, K, N, 0, 0, 1, K, 0, 1, K, 0), DeviceOp.linear(0, 1, 2, 0, 1, N, K, abi.W_F32)]
    h = cuda_backend.compile_program(DeviceProgram(ops, [N, K, N * K, N * K]))
    assert cuda_backend.program_stats(h)["early_weight_linears"] == 0
    for seed in range(6):
        W, got = np.random.default_rng(seed).standard_normal((N, K)).astype(np.float32), np.zeros(N, np.float32)
        cuda_backend.execute_program(h, [ProgramIO(1, x), ProgramIO(3, W.ravel())], [ProgramIO(0, got)])
        want, mag = W.astype(np.float64) @ x, np.abs(W).astype(np.float64) @ np.abs(x)
        assert (np.abs(got - want) <= 100 * 2.0 ** -24 * mag).all(), seed
    cuda_backend.free_program(h)


def test_which_weights_may_be_read_early(cuda_backend):
    """Those whose memory no op writes, as the LINEAR's buffer or as another one over it.  (Only the decision is looked at: ops on different buffers have no order of their own.)"""
    from zgml_b200 import DeviceBuffer, DeviceOp, DeviceProgram, ExternBuffer, abi
    N, K = 64, 512
    place = DeviceBuffer(cuda_backend, 4 * N * K)
    write, read = (DeviceOp.slice_assign(b, 3, K, N, 0, 0, 1, K, 0, 1, K, 0) for b in (2, 4)), DeviceOp.linear(0, 1, 2, 0, 1, N, K, abi.W_F32)
    for ops, early in (([read], 1), ([next(write), read], 0), ([next(write), read], 0), ([read, read], 2)):
        h = cuda_backend.compile_program(DeviceProgram(ops, [N, K, N * K, N * K, N * K], [], [], [ExternBuffer(2, place), ExternBuffer(4, place)]))
        assert cuda_backend.program_stats(h)["early_weight_linears"] == early
        cuda_backend.free_program(h)
    place.free()
