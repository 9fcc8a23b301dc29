"""MOE_FFN over bfloat16 weights with more than 16 (token, choice) pairs (experts' products on the tensor cores) against float64: runs of one row, of whole
and partial multiples of 16, at and past the most rows of a run (64 where tiles are few, 256 in the last case), experts without a row, pairs that no expert takes, widths that end within the 64-wide
steps and the 128-wide tiles.

The reference rounds what the kernels round (inputs and the activated products to bfloat16) and is float64 otherwise.  Where an f32 sum falls on the other
side of a rounding boundary of an activated product, that product is 2^-8 of itself off; the share of such values is small, so the bound is a quarter of
what all of them at once would make: 1e-3 of the output's largest value."""
import numpy as np
import pytest

from test_gpu_recops import run

pytestmark = pytest.mark.gpu


def bf16(x):
    """Round to nearest even, kept as float64."""
    u = np.asarray(x, np.float32).view(np.uint32)
    return ((u + 0x7FFF + ((u >> 16) & 1)) & np.uint32(0xFFFF0000)).view(np.float32).astype(np.float64)


@pytest.mark.parametrize("counts,top,D,ff", [([17], 1, 64, 64), ([0, 1, 16, 0, 40], 1, 72, 136), ([31, 32, 33], 1, 128, 200), ([256, 0, 257], 1, 200, 64), ([513, 15], 1, 64, 128),
                                             ([300, 20, 270], 2, 136, 264), ([5, 6, 7], 1, 1032, 72), ([100, 28], 2, 64, 1000), ([300, 0, 257, 256, 1, 16, 17, 49], 1, 64, 2432)])
def test_expert_products(cuda_backend, counts, top, D, ff):
    from zgml_b200 import DeviceBuffer, DeviceOp, ExternBuffer, abi
    from zgml_b200.backend import seq_scratch_elems
    r = np.random.default_rng(len(counts) + D)
    E, loose = len(counts), 3                                         # `loose` pairs name no expert: their token's own row counts
    pairs = sum(counts) + loose
    pairs += -pairs % top
    T = pairs // top
    chosen = np.concatenate([np.full(c, e) for e, c in enumerate(counts)] + [np.full(pairs - sum(counts), E)]).astype(np.int32)
    chosen = r.permutation(chosen)
    share = r.random(pairs).astype(np.float32)
    route = np.stack([chosen.view(np.float32), share], 1)
    x = r.standard_normal((T, D)).astype(np.float32)
    gate, up, down = (bf16(r.standard_normal((E, n, k)) / np.sqrt(k)) for n, k in ((ff, D), (ff, D), (D, ff)))
    limit, alpha, offset = 1.5, 1.2, 0.25
    words = np.concatenate([(w.astype(np.float32).view(np.uint32) >> 16).astype(np.uint16).ravel() for w in (gate, up, down)])
    w = DeviceBuffer(cuda_backend, words.nbytes, zero=False)
    w.upload(words.view(np.float32))
    op = DeviceOp.moe_ffn(0, 1, 2, 3, 4, 0, gate.size, gate.size + up.size, T, D, ff, E, top, abi.W_BF16, limit, alpha, up_offset=offset)
    got = run(cuda_backend, [op], [T * D, x.size, route.size, w.elems, seq_scratch_elems(op)], [(1, x), (2, route)], 0, (T, D), [ExternBuffer(3, w)])
    w.free()
    want = np.zeros((T, D))
    for i in range(pairs):
        e, t = chosen[i], i // top
        if e == E:
            want[t] += share[i] * x[t].astype(np.float64)
            continue
        g, u = gate[e] @ bf16(x[t]), up[e] @ bf16(x[t])
        g, u = np.minimum(g, limit), np.clip(u, -limit, limit)
        want[t] += share[i] * (down[e] @ bf16(g / (1 + np.exp(-alpha * g)) * (u + offset)))
    assert np.abs(got - want).max() < 1e-3 * np.abs(want).max()
