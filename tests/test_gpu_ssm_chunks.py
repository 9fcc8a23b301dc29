"""SSM_SCAN steps of 128 and more tokens (chunks of 64) against float64 token by token: steps that end at every kind of place in a chunk, state rows and
columns on and off the tiles, groups, constant decays, decays from almost none to one that empties the state within a token, a state slot other than the
first and a step long enough for two passes, each followed by one token that decodes from the state the step left.

Tolerance: f32 sums of up to 512 + 64 terms, in runs of 16, of products of three f32 factors: 3e-6 of the output's largest value is several times the
random sum of their roundings.  A decay near 1, rounded to f32, is off by up to 2^-25, and a state gathered over T tokens carries T of those (any f32
evaluation has that)."""
import numpy as np
import pytest

from test_gpu_recops import ctl_words, run, weights

pytestmark = pytest.mark.gpu


def step(be, state, slot, pos, xbc, dt, w, offs, H, G, N, P, constant):
    from zgml_b200 import DeviceOp, ExternBuffer, abi
    T = len(xbc)
    o = (0, H * P, H * P + G * N)
    if constant:
        op = DeviceOp.ssm_scan(0, 1, 2, None, 3, 4, *o, 0, 0, 0, 0, T, H, G, N, P, xbc.shape[1], 0, abi.W_F32, constant_decay=True)
        return run(be, [op], [T * H * P, xbc.size, H, state.elems, 8], [(1, xbc), (2, dt), (4, ctl_words(pos, slot))], 0, (T, H, P), [ExternBuffer(3, state)])
    op = DeviceOp.ssm_scan(0, 1, 2, 3, 4, 5, *o, 0, *offs, T, H, G, N, P, xbc.shape[1], H, abi.W_F32)
    return run(be, [op], [T * H * P, xbc.size, dt.size, w.elems, state.elems, 8], [(1, xbc), (2, dt), (5, ctl_words(pos, slot))], 0, (T, H, P), [ExternBuffer(3, w), ExternBuffer(4, state)])


def reference(xbc, dt, a_log, bias, skip, H, G, N, P, constant):
    import torch
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda().double()
    z, n = d(xbc), len(xbc)
    x = z[:, :H * P].view(n, H, P)
    B, C = (z[:, H * P + i * G * N:H * P + (i + 1) * G * N].view(n, G, N).repeat_interleave(H // G, 1) for i in (0, 1))
    if constant:
        dec, st, sk = d(dt).expand(n, H), torch.ones(n, H, dtype=torch.float64, device="cuda"), torch.zeros(H, dtype=torch.float64, device="cuda")
    else:
        st = torch.nn.functional.softplus(d(dt) + d(bias))
        dec, sk = torch.exp(-d(a_log).exp() * st), d(skip)
    S, out = torch.zeros(H, N, P, dtype=torch.float64, device="cuda"), torch.empty(n, H, P, dtype=torch.float64, device="cuda")
    for t in range(n):
        S = dec[t][:, None, None] * S + (st[t][:, None] * B[t])[:, :, None] * x[t][:, None, :]
        out[t] = torch.einsum("hnp,hn->hp", S, C[t]) + sk[:, None] * x[t]
    return out.cpu().numpy()


CASES = [(128, 2, 1, 4, 4), (129, 2, 2, 32, 32), (191, 4, 2, 36, 36), (192, 1, 1, 64, 64), (193, 3, 1, 68, 68), (255, 2, 1, 128, 132), (320, 2, 2, 132, 8), (130, 1, 1, 512, 64), (1027, 2, 1, 16, 100),
         (700, 40, 1, 64, 64), (300, 80, 2, 512, 128)]


@pytest.mark.parametrize("T,H,G,N,P", CASES)
@pytest.mark.parametrize("rate", ["slow", "usual", "fast", "constant"])
def test_ssm_scan_by_chunks(cuda_backend, T, H, G, N, P, rate):
    from zgml_b200 import DeviceBuffer, DeviceOp, abi
    from zgml_b200.backend import seq_state_elems
    if (T, H) == (300, 80) and rate not in ("usual", "constant"):
        pytest.skip("two passes: one rate of either form")
    r = np.random.default_rng(T + N)
    constant = rate == "constant"
    n = T + 1
    xbc = r.standard_normal((n, H * P + 2 * G * N)).astype(np.float32)
    xbc[:, H * P:] *= N ** -0.25
    a_log = (r.random(H) + {"slow": -9.0, "usual": -1.0, "fast": 5.0, "constant": 0.0}[rate]).astype(np.float32)
    bias, skip = (r.standard_normal(H) - 1.0).astype(np.float32), r.standard_normal(H).astype(np.float32)
    dt = r.uniform(0.5, 1.0, H).astype(np.float32) if constant else r.standard_normal((n, H)).astype(np.float32)
    w, offs = weights(cuda_backend, a_log, bias, skip)
    probe = DeviceOp.ssm_scan(0, 1, 2, 3, 4, 5, 0, H * P, H * P + G * N, 0, *offs, T, H, G, N, P, xbc.shape[1], H, abi.W_F32)
    state = DeviceBuffer(cuda_backend, 4 * 2 * seq_state_elems(probe))
    got = [step(cuda_backend, state, 1, at, xbc[at:at + m], dt if constant else dt[at:at + m], w, offs, H, G, N, P, constant) for at, m in ((0, T), (T, 1))]
    state.free()
    w.free()
    want = reference(xbc, dt, a_log, bias, skip, H, G, N, P, constant)
    assert np.abs(np.concatenate(got) - want).max() < (3e-6 + (0 if constant else T * 2.0 ** -25)) * np.abs(want).max()


@pytest.mark.parametrize("at", [64, 70, 100, 127])
def test_an_input_that_is_no_number_spares_the_tokens_before_it(cuda_backend, at):
    from zgml_b200 import DeviceBuffer, DeviceOp, abi
    from zgml_b200.backend import seq_state_elems
    r = np.random.default_rng(3)
    T, H, G, N, P = 140, 2, 1, 32, 32
    xbc, dt = r.standard_normal((T, H * P + 2 * G * N)).astype(np.float32), r.standard_normal((T, H)).astype(np.float32)
    w, offs = weights(cuda_backend, r.standard_normal(H), r.standard_normal(H), r.standard_normal(H))
    probe = DeviceOp.ssm_scan(0, 1, 2, 3, 4, 5, 0, H * P, H * P + G * N, 0, *offs, T, H, G, N, P, xbc.shape[1], H, abi.W_F32)
    outs = []
    for bad in (0.0, np.inf, np.nan):
        xbc[at, 3] = bad
        state = DeviceBuffer(cuda_backend, 4 * seq_state_elems(probe))
        outs.append(step(cuda_backend, state, 0, 0, xbc, dt, w, offs, H, G, N, P, False))
        state.free()
    w.free()
    for out in outs[1:]:
        assert np.abs(out[:at] - outs[0][:at]).max() < 1e-6 * np.abs(outs[0][:at]).max() and not np.isfinite(out[at, 0, 3]) and np.isfinite(out[:, :, 4:]).all()


def test_chunks_are_no_further_off_than_the_walk(cuda_backend):
    """The same 1024 tokens in one step (chunks of 64) and in steps of 64 (token by token), four random inputs of 16 heads: distances from float64, whose sum over
    the inputs may not be larger by chunks (3 % for the draw of the roundings; with C . B as f32 chains of 32 terms it was 11 % larger)."""
    from zgml_b200 import DeviceBuffer, DeviceOp, abi
    from zgml_b200.backend import seq_state_elems
    T, H, G, N, P = 1024, 16, 1, 128, 64
    off = {1024: 0.0, 64: 0.0}
    for seed in range(4):
        r = np.random.default_rng(100 + seed)
        xbc, dt = (0.6 * r.standard_normal((T, H * P + 2 * N))).astype(np.float32), r.standard_normal((T, H)).astype(np.float32)
        a_log, bias, skip = (a.astype(np.float32) for a in (np.log(1 + 15 * r.random(H)), r.uniform(-5, -1, H), r.uniform(0.5, 1.5, H)))
        w, offs = weights(cuda_backend, a_log, bias, skip)
        want = reference(xbc, dt, a_log, bias, skip, H, G, N, P, False)
        probe = DeviceOp.ssm_scan(0, 1, 2, 3, 4, 5, 0, H * P, H * P + G * N, 0, *offs, T, H, G, N, P, xbc.shape[1], H, abi.W_F32)
        for n in off:
            state = DeviceBuffer(cuda_backend, 4 * seq_state_elems(probe))
            got = np.concatenate([step(cuda_backend, state, 0, at, xbc[at:at + n], dt[at:at + n], w, offs, H, G, N, P, False) for at in range(0, T, n)])
            state.free()
            off[n] += np.linalg.norm(got - want) / np.linalg.norm(want)
        w.free()
    assert off[1024] <= 1.03 * off[64]
