"""CACHED_ATTENTION with at most 16 rows (operands cut into three bfloat16 parts, mma.sync) against float64: key dimensions and value widths around the 16s and
32s that an operand holds, one to 16 rows, key counts around the 32 of a buffer and the shares, every width of CTA, and values that are not finite or round to infinity as bfloat16.

Tolerance: the parts keep all 24 bits of an operand and the products left out are below 2^-23 of a term; scores of up to about 10 are then off by a few 2^-23 of that
and f32 sums of up to a few thousand terms add as much: 1e-5 of the output's scale is more than five times what that comes to."""
import numpy as np
import pytest

from test_gpu_attention_tc import case, close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,pos,H,G,dk,dv,kw", [
    (1, 0, 4, 4, 4, 4, {}),
    (1, 30, 8, 1, 16, 32, {}),
    (1, 31, 8, 1, 20, 36, {}),
    (1, 32, 16, 1, 32, 64, {}),
    (2, 62, 8, 1, 44, 68, {}),
    (16, 63, 3, 3, 72, 128, {}),
    (5, 100, 6, 2, 132, 132, dict(sink=True)),
    (3, 700, 10, 2, 192, 256, dict(cap=20.0)),
    (1, 2111, 16, 1, 64, 64, dict(slot=1)),
    (1, 4095, 4, 1, 576, 260, {}),
    (4, 4095, 2, 2, 64, 512, dict(maps=2, out_scale=0.5)),
    (1, 300, 2, 1, 36, 640, dict(table=True)),
    (1, 300, 16, 1, 256, 1024, dict(sigmoid=True, table=True)),
    (7, 9, 2, 1, 64, 64, dict(mask="window", size=6)),
    (9, 3000, 4, 4, 96, 96, dict(mask="window", size=513, R=530)),
    (3, 200, 4, 2, 128, 128, dict(mask="block", size=64, gain=1e18)),
    (2, 129, 8, 2, 128, 64, dict(gain=1e-18)),
    (1, 2100, 8, 8, 60, 64, {}),                       # more CTAs than SMs: four and eight warps; few: eight and sixteen
    (3, 2100, 12, 4, 64, 68, {}),
    (2, 2100, 6, 6, 36, 256, {}),
    (2, 70, 16, 2, 36, 256, {}),
    (5, 40, 6, 2, 68, 100, {}),
])
def test_few_rows(cuda_backend, T, pos, H, G, dk, dv, kw):
    got, want, _, _ = case(cuda_backend, T, pos, H, G, dk, dv, seed=T + pos + dk, **kw)
    assert close(got, want)


@pytest.mark.parametrize("dk,dv", [(64, 64), (128, 192), (320, 512)])
@pytest.mark.parametrize("where,value", [("k", np.inf), ("v", np.inf), ("v", -np.inf), ("v", np.nan), ("v", 3.4e38)])
def test_not_finite(cuda_backend, dk, dv, where, value):
    def poison(k, v):
        (k if where == "k" else v)[1500, 3] = value      # seen by the only row of each head; head 0's columns
    got, want, _, _ = case(cuda_backend, 1, 2000, 8, 4, dk, dv, seed=dk, poison=poison)
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isposinf(got), np.isposinf(want)) and np.array_equal(np.isneginf(got), np.isneginf(want))
    fine = np.isfinite(want) & (np.abs(want) < 1e30)
    assert np.abs(got - want)[fine].max() <= 1e-5 * np.abs(want[fine]).max()
    big = np.isfinite(want) & ~fine
    assert np.allclose(got[big], want[big], rtol=1e-5)
