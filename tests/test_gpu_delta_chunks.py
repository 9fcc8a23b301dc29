"""DELTA_RULE in chunks of 16 tokens where the launches differ: steps walked in several passes of prepared vectors, more CTAs than SMs (two stages of
shared memory instead of three), one stage (512 key rows), chunks that end one token early, on time and one late; and short steps, by blocks of four tokens.

Tolerance: as for the shorter steps, sums of at most 512 f32 terms of a state that the decay keeps at the inputs' size: a few 1e-6 of the output's largest
value, 2e-5 with room for the normalisation's division by a small root."""
import numpy as np
import pytest

from test_gpu_gateops import _rule_reference, weights
from test_gpu_recops import ctl_words, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,H,dim,vdim", [(1320, 8, 512, 16), (47, 80, 64, 40), (65, 80, 64, 40), (48, 75, 128, 32), (49, 3, 256, 20), (63, 1, 512, 7)],
                         ids=["two passes", "two stages, 47 tokens by blocks", "two stages, 64 rows", "two stages, 128 rows", "256 rows", "one stage"])
@pytest.mark.parametrize("plain", [False, True], ids=["corrected", "plain"])
def test_delta_rule_in_chunks(cuda_backend, plain, T, H, dim, vdim):
    step(cuda_backend, plain, T, H, dim, vdim)


def step(cuda_backend, plain, T, H, dim, vdim):
    from zgml_b200 import DeviceBuffer, DeviceOp, ExternBuffer, abi
    r = np.random.default_rng(T)
    eps, unit_eps, q_scale = 1e-5, 1e-6, 0.4
    qrs = 2 * H * dim + 2 * H * vdim + H
    A_log, dt_bias, norm_w = r.standard_normal(H) * 0.5, r.standard_normal((H, dim)) * 0.5 - 1.0, 1 + 0.2 * r.standard_normal(vdim)
    w, (oA, odt, onw) = weights(cuda_backend, A_log, dt_bias, norm_w)
    state = DeviceBuffer(cuda_backend, 4 * H * dim * vdim)
    proj = r.standard_normal((T, qrs)).astype(np.float32)
    proj[:, :2 * H * dim] *= dim ** -0.5
    a = r.standard_normal((T, H * dim)).astype(np.float32)
    q, k = proj[:, :H * dim].reshape(T, H, dim), proj[:, H * dim:2 * H * dim].reshape(T, H, dim)
    v, gate = proj[:, 2 * H * dim:2 * H * dim + H * vdim].reshape(T, H, vdim), proj[:, 2 * H * dim + H * vdim:2 * H * dim + 2 * H * vdim].reshape(T, H, vdim)
    beta = proj[:, 2 * H * dim + 2 * H * vdim:]
    op = DeviceOp.delta_rule(0, 1, None if plain else 1, 2, 1, 3, 4, 5, 0, H * dim, 2 * H * dim, 2 * H * dim + 2 * H * vdim, oA, odt, onw, T, H, H, dim, vdim, qrs, qrs,
                             H * dim, qrs, abi.W_F32, eps, unit_eps, q_scale, gate_off=2 * H * dim + H * vdim, plain=plain)
    got = run(cuda_backend, [op], [T * H * vdim, proj.size, a.size, w.elems, state.elems, 8], [(1, proj), (2, a), (5, ctl_words(0, 0))], 0, (T, H, vdim),
              [ExternBuffer(3, w), ExternBuffer(4, state)])
    f64 = lambda x: x.astype(np.float64)  # noqa: E731
    want, S_want = _rule_reference(dict(plain=plain, sigmoid_decay=False, silu_gate=False), np.zeros((H, dim, vdim)), f64(q), f64(k), f64(v), f64(beta), f64(a).reshape(T, H, dim),
                                   f64(gate), f64(np.float32(A_log)), f64(np.float32(dt_bias)), f64(np.float32(norm_w)), 1.0, q_scale, eps, unit_eps, 1.0)
    assert np.abs(got - want).max() < 2e-5 * max(1.0, np.abs(want).max())
    S_got = state.download(np.float32, 0, H * dim * vdim).reshape(H, dim, vdim)
    assert np.abs(S_got - S_want).max() < 2e-5 * max(1.0, np.abs(S_want).max())
    w.free()
    state.free()


@pytest.mark.parametrize("T,H,dim,vdim", [(16, 1, 5, 3), (31, 3, 64, 17), (32, 3, 64, 17), (39, 2, 32, 9), (40, 2, 32, 9), (52, 16, 33, 64), (53, 16, 33, 64), (41, 150, 20, 24),
                                          (16, 12, 128, 128), (23, 10, 97, 128), (23, 11, 97, 128), (24, 18, 65, 120), (25, 18, 65, 120), (24, 9, 128, 128), (17, 20, 128, 128)])
@pytest.mark.parametrize("plain", [False, True], ids=["corrected", "plain"])
def test_short_steps_on_both_sides_of_the_rule(cuda_backend, plain, T, H, dim, vdim):
    """Steps of blocks of four tokens, with two and four key rows per lane, and the next ones that go by chunks."""
    step(cuda_backend, plain, T, H, dim, vdim)


@pytest.mark.parametrize("dim,vdim", [(64, 64), (100, 20), (256, 16), (512, 7)])
@pytest.mark.parametrize("plain,value", [(True, 3.4e38), (False, 3.4e38), (True, np.inf)], ids=["plain", "corrected", "plain, infinite"])
def test_magnitudes_beyond_bfloat16(cuda_backend, plain, value, dim, vdim):
    """A value of token 20, or an element of the state before the step, lies between bfloat16's largest number and f32's, or is infinite: what is a number stays one, and
    every column is within the tolerance of its own largest element.  (The queries are scaled so that the squares of the outputs stay in range.)"""
    from zgml_b200 import DeviceBuffer, DeviceOp, ExternBuffer, abi
    r = np.random.default_rng(dim)
    T, H, eps, unit_eps, q_scale = 70, 2, 1e-5, 1e-6, 1e-25
    qrs = 2 * H * dim + 2 * H * vdim + H
    A_log, dt_bias, norm_w = r.standard_normal(H) * 0.5, r.standard_normal((H, dim)) * 0.5 - 5.0, 1 + 0.2 * r.standard_normal(vdim)
    w, (oA, odt, onw) = weights(cuda_backend, A_log, dt_bias, norm_w)
    proj, a = r.standard_normal((T, qrs)).astype(np.float32), r.standard_normal((T, H * dim)).astype(np.float32)
    proj[:, :2 * H * dim] *= dim ** -0.5
    S = r.standard_normal((H, dim, vdim)).astype(np.float32)
    if plain:
        proj[20, 2 * H * dim + 3] = value
    else:
        S[0, 5, 2] = value
    state = DeviceBuffer(cuda_backend, S.nbytes, zero=False)
    state.upload(S.ravel())
    q, k = proj[:, :H * dim].reshape(T, H, dim), proj[:, H * dim:2 * H * dim].reshape(T, H, dim)
    v, gate = proj[:, 2 * H * dim:2 * H * dim + H * vdim].reshape(T, H, vdim), proj[:, 2 * H * dim + H * vdim:2 * H * dim + 2 * H * vdim].reshape(T, H, vdim)
    beta = proj[:, 2 * H * dim + 2 * H * vdim:]
    op = DeviceOp.delta_rule(0, 1, None if plain else 1, 2, 1, 3, 4, 5, 0, H * dim, 2 * H * dim, 2 * H * dim + 2 * H * vdim, oA, odt, onw, T, H, H, dim, vdim, qrs, qrs,
                             H * dim, qrs, abi.W_F32, eps, unit_eps, q_scale, gate_off=2 * H * dim + H * vdim, plain=plain)
    got = run(cuda_backend, [op], [T * H * vdim, proj.size, a.size, w.elems, state.elems, 8], [(1, proj), (2, a), (5, ctl_words(0, 0))], 0, (T, H, vdim),
              [ExternBuffer(3, w), ExternBuffer(4, state)])
    f64 = lambda x: x.astype(np.float64)  # noqa: E731
    with np.errstate(all="ignore"):
        want, S_want = _rule_reference(dict(plain=plain, sigmoid_decay=False, silu_gate=False), f64(S), f64(q), f64(k), f64(v), f64(beta), f64(a).reshape(T, H, dim),
                                       f64(gate), f64(np.float32(A_log)), f64(np.float32(dt_bias)), f64(np.float32(norm_w)), 1.0, q_scale, eps, unit_eps, 1.0)
    S_got = state.download(np.float32, 0, H * dim * vdim).reshape(H, dim, vdim)
    fine = np.isfinite(want)
    if np.isinf(value):
        assert not np.isfinite(got[20:, 0]).all(1).any()      # (which of a row's outputs are infinite and which are no numbers is left open)
    else:
        assert fine.all()
    assert np.abs(got - want)[fine].max() < 2e-5 * max(1.0, np.abs(want[fine]).max())
    assert np.array_equal(np.isposinf(S_got), np.isposinf(S_want)) and np.array_equal(np.isneginf(S_got), np.isneginf(S_want))
    for h in range(H):
        for c in range(vdim):
            if np.isfinite(S_want[h, :, c]).all():
                assert np.abs(S_got[h, :, c] - S_want[h, :, c]).max() < 2e-5 * np.abs(S_want[h, :, c]).max(), (h, c)
    w.free()
    state.free()
