"""The streamed matvec where a column group's chunk count has no divisor near the chunks of a CTA (pieces of one size and a shorter last one), against the
oracle at the bar of test_gpu_qgemv_stream.py: prime counts of both chunk sizes, a last piece of one chunk, pieces longer than a staging segment."""
import numpy as np
import pytest

from test_gpu_qgemv_stream import _forced_backend, _weights
from test_gpu_qmatmul import oracle_out, rel_err, rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunks,K,N", [(3, 448, 96), (3, 32 * 22 - 7, 64), (4, 32 * 4 * 7, 288), (16, 32 * 361, 96), (16, 32 * 277, 320), (32, 32 * 2 * 67, 64), (70, 32 * 2 * 151, 32), (66, 32 * 4 * 139, 32)])
@pytest.mark.parametrize("kind", ["i8_f32", "q8_0", "q4_0"])
def test_uneven_pieces(chunks, K, N, kind):
    be = _forced_backend(chunks)
    K -= K % (1 if kind == "i8_f32" else 32)
    o, up = _weights(kind, K, N, 5 + K + N)
    w = up(be)
    x = rng(K).standard_normal((1, K)).astype(np.float32)
    outs = [w.matmul(x, 1) for _ in range(3)]
    w.free()
    be.close()
    assert rel_err(outs[0], oracle_out(o, x, 1)) < 2e-5
    assert all(np.array_equal(g.view(np.uint32), outs[0].view(np.uint32)) for g in outs[1:])
