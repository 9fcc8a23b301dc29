"""DELTA_RULE steps of 16 and more tokens (four tokens at a time) against float64: steps that end at every place of a block and of a staged tile, key
dimensions and value widths on and off the 32 rows per lane slot and the 16 columns of a CTA, three decays (none to speak of, ordinary, and one that
wipes the state within a block).

Tolerance: the sums have at most 512 terms, in f32, of a state that the decay keeps at the inputs' size: a few 1e-6 of the output's largest value; 2e-5
leaves room for the normalisation's division by a small root."""
import numpy as np
import pytest

from test_gpu_gateops import _rule_reference, weights
from test_gpu_recops import ctl_words, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("decay", [-8.0, 0.0, 30.0])
@pytest.mark.parametrize("T,dim,vdim", [(16, 32, 16), (17, 33, 1), (18, 64, 17), (19, 65, 31), (20, 96, 32), (31, 128, 48), (32, 129, 5), (33, 256, 15), (67, 257, 33), (21, 512, 18)])
@pytest.mark.parametrize("plain", [False, True], ids=["corrected", "plain"])
def test_delta_rule_in_blocks_of_four(cuda_backend, plain, T, dim, vdim, decay):
    from zgml_b200 import DeviceBuffer, DeviceOp, ExternBuffer, abi
    r = np.random.default_rng(T)
    H, eps, unit_eps, q_scale = 2, 1e-5, 1e-6, 0.4
    qrs = 2 * H * dim + 2 * H * vdim + H
    A_log, dt_bias, norm_w = r.standard_normal(H) * 0.5, r.standard_normal((H, dim)) * 0.5 + decay, 1 + 0.2 * r.standard_normal(vdim)
    w, (oA, odt, onw) = weights(cuda_backend, A_log, dt_bias, norm_w)
    state = DeviceBuffer(cuda_backend, 4 * H * dim * vdim)
    S_want = np.zeros((H, dim, vdim))
    form = dict(plain=plain, sigmoid_decay=False, silu_gate=False)
    for rep in range(2):                                              # the second step starts from a state
        proj = r.standard_normal((T, qrs)).astype(np.float32)
        proj[:, :2 * H * dim] *= dim ** -0.5
        a = r.standard_normal((T, H * dim)).astype(np.float32)
        q, k = proj[:, :H * dim].reshape(T, H, dim), proj[:, H * dim:2 * H * dim].reshape(T, H, dim)
        v, gate = proj[:, 2 * H * dim:2 * H * dim + H * vdim].reshape(T, H, vdim), proj[:, 2 * H * dim + H * vdim:2 * H * dim + 2 * H * vdim].reshape(T, H, vdim)
        beta = proj[:, 2 * H * dim + 2 * H * vdim:]
        op = DeviceOp.delta_rule(0, 1, None if plain else 1, 2, 1, 3, 4, 5, 0, H * dim, 2 * H * dim, 2 * H * dim + 2 * H * vdim, oA, odt, onw, T, H, H, dim, vdim, qrs, qrs,
                                 H * dim, qrs, abi.W_F32, eps, unit_eps, q_scale, gate_off=2 * H * dim + H * vdim, plain=plain)
        got = run(cuda_backend, [op], [T * H * vdim, proj.size, a.size, w.elems, state.elems, 8], [(1, proj), (2, a), (5, ctl_words(rep * T, 0))], 0, (T, H, vdim),
                  [ExternBuffer(3, w), ExternBuffer(4, state)])
        f64 = lambda x: x.astype(np.float64)
        want, S_want = _rule_reference(form, S_want, f64(q), f64(k), f64(v), f64(beta), f64(a).reshape(T, H, dim), f64(gate), f64(np.float32(A_log)), f64(np.float32(dt_bias)),
                                       f64(np.float32(norm_w)), 1.0, q_scale, eps, unit_eps, 1.0)
        assert np.abs(got - want).max() < 2e-5 * max(1.0, np.abs(want).max()), rep
        S_got = state.download(np.float32, 0, H * dim * vdim).reshape(H, dim, vdim)
        assert np.abs(S_got - S_want).max() < 2e-5 * max(1.0, np.abs(S_want).max()), rep
    w.free()
    state.free()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_a_value_that_is_no_number_spares_the_tokens_before_it(cuda_backend, bad):
    """The value of token 18 (the third of its block) is not finite: the tokens before it come out as without it."""
    from zgml_b200 import DeviceBuffer, DeviceOp, ExternBuffer, abi
    r = np.random.default_rng(5)
    T, H, dim, vdim = 20, 1, 32, 16
    w, (oA, odt, onw) = weights(cuda_backend, r.standard_normal(H), r.standard_normal((H, dim)), 1 + 0.2 * r.standard_normal(vdim))
    qrs = 2 * dim + 2 * vdim + H
    proj, a = r.standard_normal((T, qrs)).astype(np.float32), r.standard_normal((T, dim)).astype(np.float32)
    outs = []
    for value in (0.5, bad):
        proj[18, 2 * dim:2 * dim + vdim] = value
        state = DeviceBuffer(cuda_backend, 4 * dim * vdim)
        op = DeviceOp.delta_rule(0, 1, 1, 2, 1, 3, 4, 5, 0, dim, 2 * dim, 2 * dim + 2 * vdim, oA, odt, onw, T, H, H, dim, vdim, qrs, qrs, dim, qrs, abi.W_F32, 1e-5, 1e-6, 0.4, gate_off=2 * dim + vdim)
        outs.append(run(cuda_backend, [op], [T * vdim, proj.size, a.size, w.elems, state.elems, 8], [(1, proj), (2, a), (5, ctl_words(0, 0))], 0, (T, vdim), [ExternBuffer(3, w), ExternBuffer(4, state)]))
        state.free()
    w.free()
    assert np.array_equal(outs[0][:18], outs[1][:18]) and not np.isfinite(outs[1][18]).any()
