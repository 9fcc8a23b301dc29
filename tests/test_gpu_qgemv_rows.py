"""Quantized matmuls of three to eight rows against the oracle: k-ranges of less than a record per warp, of up to 64 records (two teams of warps) and one more, of
a warp's eight records and one more (K split over a cluster of two and four CTAs, over three by global scratch), rows past the end of K, column groups whose scales
differ by powers of two, more column groups than wait for a cluster, and rows that are not finite.

The bar is the matvec's: 2e-5 of the largest output (a 23-bit grid relative to the largest activation of a warp's 256)."""
import numpy as np
import pytest

from test_gpu_qgemv_stream import _weights
from test_gpu_qmatmul import oracle_out, rel_err, rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K,N", [(3, 32, 32), (8, 32, 4800), (5, 480, 96), (4, 2048, 4800), (8, 2080, 4800), (6, 4096, 160), (7, 4128, 64), (8, 9000, 1024), (3, 14336, 3200), (8, 16384, 64)])
@pytest.mark.parametrize("kind", ["i8_f32", "q8_0", "q4_0"])
def test_rows_in_one_pass(cuda_backend, kind, M, K, N):
    K -= K % (1 if kind == "i8_f32" else 32)
    o, up = _weights(kind, K, N, K + N)
    w = up(cuda_backend)
    x = rng(K).standard_normal((M, K)).astype(np.float32) * np.float32(2.0) ** np.arange(-3, M - 3, dtype=np.float32)[:, None]
    outs = [w.matmul(x, M) for _ in range(2)]
    want = oracle_out(o, x, M)
    for m in range(M):
        assert rel_err(outs[0][m], want[m]) < 2e-5, m
    assert np.array_equal(outs[0].view(np.uint32), outs[1].view(np.uint32))
    x[1, K // 2] = np.inf
    bad = w.matmul(x, M)
    assert not np.isfinite(bad[1]).any() and np.array_equal(bad[[0, 2]], outs[0][[0, 2]])
    w.free()


def test_column_groups_of_different_scales(cuda_backend):
    from zgml_b200 import QuantizedWeight
    r, K, N, M = rng(9), 192, 320, 5
    q = r.integers(-127, 128, (K, N)).astype(np.int8)
    s = (r.uniform(0.5, 1.0, (K, N // 32)) * 2.0 ** (3 * (np.arange(N // 32) % 4))).astype(np.float32)
    w = QuantizedWeight.upload(cuda_backend, q.reshape(-1), s.reshape(-1), K, N)
    x = r.standard_normal((M, K)).astype(np.float32)
    got, want = w.matmul(x, M), x.astype(np.float64) @ (q * np.repeat(s, 32, 1).astype(np.float64))
    for n in range(0, N, 32):
        assert rel_err(got[:, n:n + 32], want[:, n:n + 32]) < 2e-5, n
    w.free()


@pytest.mark.parametrize("M", [1, 2, 5])
def test_matvecs_of_unequal_widths_share_a_launch(cuda_backend, M):
    """q, k and v of grouped heads: one K, two widths, one launch; the outputs are those of the matvecs alone."""
    from zgml_b200 import DeviceOp, DeviceProgram, ProgramIO
    from zgml_b200.backend import ResidentQuantizedWeight
    K, widths = 576, (192, 576, 192, 64)
    ws = [_weights("q8_0", K, N, N + 1)[1](cuda_backend) for N in widths]
    x = rng(M).standard_normal((M, K)).astype(np.float32)
    ops = [DeviceOp.qmatmul(1 + i, 0, i, M, N, K) for i, N in enumerate(widths)]
    h = cuda_backend.compile_program(DeviceProgram(ops, [M * K] + [M * N for N in widths], [], [ResidentQuantizedWeight(w) for w in ws]))
    got = [np.zeros((M, N), np.float32) for N in widths]
    cuda_backend.execute_program(h, [ProgramIO(0, x.ravel())], [ProgramIO(1 + i, g) for i, g in enumerate(got)])
    for w, g in zip(ws, got):
        assert np.array_equal(g, w.matmul(x, M))
    cuda_backend.free_program(h)
    for w in ws:
        w.free()
