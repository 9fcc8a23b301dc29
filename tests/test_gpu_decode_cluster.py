"""The layers of a small single-token LLaMA on one thread-block cluster (csrc/decode_cluster.cu) against the general schedule of the same program (which the other LLaMA
tests hold against the oracle): every program buffer, at the edges of what the kernel splits — head widths, query heads per KV head, KV heads that do not divide the CTAs,
column groups and feed-forward pairs that do not either, positions around a stage of keys and past all of them, other activations; and what the form is taken for."""
import os

import numpy as np
import pytest

from zgml_b200.host.llama import DeviceLlamaSession, LlamaConfig, synthetic_weights

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def general():
    from zgml_b200 import CudaBackend
    old = os.environ.get("ZG_CUDA_DECODE_CLUSTER")
    os.environ["ZG_CUDA_DECODE_CLUSTER"] = "0"
    try:
        return CudaBackend(0)
    finally:
        if old is None:
            os.environ.pop("ZG_CUDA_DECODE_CLUSTER")
        else:
            os.environ["ZG_CUDA_DECODE_CLUSTER"] = old


#          d_head, heads, kv, ff, max_seq
SHAPES = [(32, 1, 1, 32, 40),          # one column group, one pair: most CTAs have nothing
          (32, 3, 3, 96, 200), (32, 16, 16, 544, 330), (64, 4, 1, 256, 1100), (64, 9, 3, 1536, 700), (64, 10, 5, 800, 420), (128, 2, 2, 288, 600), (128, 2, 1, 640, 1100),
          # with the eight above: every head width with every count of query heads per KV head that the kernel is compiled for
          (32, 2, 1, 96, 300), (32, 6, 2, 160, 300), (32, 8, 2, 256, 300), (64, 3, 3, 224, 300)]


@pytest.mark.parametrize("kind", ["q8_0", "q4_0", "i8_f32"])
@pytest.mark.parametrize("dh,heads,kv,ff,seq", SHAPES)
def test_every_buffer_as_the_general_schedule_leaves_it(cuda_backend, general, dh, heads, kv, ff, seq, kind):
    from zgml_b200 import ProgramIO
    cfg = LlamaConfig(vocab_size=64, d_model=dh * heads, n_layers=3, n_heads=heads, n_kv_heads=kv, d_ff=ff, max_seq_len=seq)
    w = synthetic_weights(cfg, "q4_0" if kind == "q4_0" else "q8_0", seed=dh + heads + ff, embed_scale=1.0)
    if kind == "i8_f32":           # scales that half precision does not hold keep their 32 bits
        for layer in w.layers:
            for u in layer.values():
                u.scales[:] *= np.float32(1.0001)
    dev, ref = DeviceLlamaSession(cuda_backend, cfg, w, 1), DeviceLlamaSession(general, cfg, w, 1)
    assert cuda_backend.program_stats(dev.handle)["fused_decode_layers"] == 3 and general.program_stats(ref.handle)["fused_decode_layers"] == 0
    sizes = dev.lp.program.buffer_sizes
    got, want = ([np.zeros(n, np.float32) for n in sizes] for _ in range(2))
    dev.outputs = [ProgramIO(i, b) for i, b in enumerate(got)]
    ref.outputs = [ProgramIO(i, b) for i, b in enumerate(want)]
    for pos in [0, 1, 2, 15, 16, 31, 32, 33, 63, 64, 127, 128, 129, seq - 1]:
        if pos >= seq:
            continue
        dev.execute_at([(7 * pos + 1) % 64], pos)
        ref.execute_at([(7 * pos + 1) % 64], pos)
        for i, (g, v) in enumerate(zip(got, want)):
            fin = np.isfinite(v)
            assert np.array_equal(np.isfinite(g), fin), f"buffer {i} at position {pos}"
            # a product of K terms on a grid of 2^-24 of its largest is off by some 2^-24 sqrt(K) = 1.4e-6 of its own size; seven in a row per layer, three layers, and scores
            # of up to 10 that a softmax turns into factors: 1e-4, which is what either schedule is held to against the oracle
            assert np.max(np.abs(g[fin] - v[fin]), initial=0.0) <= 1e-4 * np.max(np.abs(v[fin]), initial=0.0) + 1e-6, f"buffer {i} at position {pos}"
    dev.close()
    ref.close()


@pytest.mark.parametrize("chain", ["gelu", "two constants", "gate and up"])
def test_other_activations(cuda_backend, general, monkeypatch, chain):
    """Chains other than SiLU run through the interpreter of steps: unary ops, constants (the first is read ahead, a second is not), gate and up as operands, either order."""
    from zgml_b200 import DeviceOp, ProgramIO, abi
    from zgml_b200.host import llama
    cfg = LlamaConfig(vocab_size=64, d_model=192, n_layers=2, n_heads=3, n_kv_heads=1, d_ff=1120, max_seq_len=24)      # 35 pairs of column groups
    w = synthetic_weights(cfg, "q8_0", seed=9, embed_scale=1.0)
    plain = llama.build_program

    def build(cfg, w, token_len=1):
        lp = plain(cfg, w, token_len)
        r, F = np.random.default_rng(4), cfg.d_ff
        first, second = (len(lp.program.buffer_sizes) + i for i in range(2))
        lp.program.buffer_sizes += [F + 8, F + 4]
        lp.program.initial_uploads += [ProgramIO(first, r.standard_normal(F + 8).astype(np.float32)), ProgramIO(second, r.standard_normal(F + 4).astype(np.float32))]
        for i, op in enumerate(lp.program.ops):
            if op.tag != abi.OP_FUSED_ELEMENTWISE:
                continue
            gate, silu, up = op.u.fused_elementwise.src, op.u.fused_elementwise.dst, lp.program.ops[i + 1].u.elementwise.src1
            steps = {"gelu": [("gelu", 0, 0, 0)], "two constants": [("abs", 0, 0, 0), ("mul", 1, first, 8), ("relu", 0, 0, 0), ("add", 0, second, 4), ("neg", 0, 0, 0)],
                     "gate and up": [("add", 1, up, 0), ("mul", 0, gate, 0), ("abs", 0, 0, 0), ("sqrt", 0, 0, 0)]}[chain]
            lp.program.ops[i] = DeviceOp.fused_elementwise(steps, F, silu, gate)
        return lp
    monkeypatch.setattr(llama, "build_program", build)
    dev, ref = DeviceLlamaSession(cuda_backend, cfg, w, 1), DeviceLlamaSession(general, cfg, w, 1)
    assert cuda_backend.program_stats(dev.handle)["fused_decode_layers"] == 2 and general.program_stats(ref.handle)["fused_decode_layers"] == 0
    got, want = ([np.zeros(n, np.float32) for n in dev.lp.program.buffer_sizes] for _ in range(2))
    dev.outputs, ref.outputs = ([ProgramIO(i, b) for i, b in enumerate(bufs)] for bufs in (got, want))
    for pos in range(3):
        dev.execute_at([pos + 1], pos)
        ref.execute_at([pos + 1], pos)
        for i, (g, v) in enumerate(zip(got, want)):
            fin = np.isfinite(v)
            assert np.array_equal(np.isfinite(g), fin) and np.max(np.abs(g[fin] - v[fin]), initial=0.0) <= 1e-4 * np.max(np.abs(v[fin]), initial=0.0) + 1e-6, f"buffer {i} at position {pos}"
    dev.close()
    ref.close()


def test_not_finite_input_comes_out_as_the_oracle_has_it(cuda_backend):
    """Positions whose score is not finite are passed over, with whatever their values hold."""
    from llama_reference import OracleBackend
    cfg = LlamaConfig(vocab_size=64, d_model=192, n_layers=2, n_heads=3, n_kv_heads=1, d_ff=256, max_seq_len=64)
    for bad in (np.nan, np.inf, 3e38, 1e-38):
        w = synthetic_weights(cfg, "q8_0", seed=3, embed_scale=1.0)
        w.token_embed[5, 17] = bad
        dev, ref = DeviceLlamaSession(cuda_backend, cfg, w, 1), DeviceLlamaSession(OracleBackend(), cfg, w, 1)
        for t in (4, 5, 6):
            a, b = dev.step(t).copy(), ref.step(t).copy()
            assert np.array_equal(np.isfinite(a), np.isfinite(b)), (bad, t)
            fin = np.isfinite(b)
            assert np.max(np.abs(a[fin] - b[fin]), initial=0.0) <= 1e-4 * np.max(np.abs(b[fin]), initial=0.0)
        dev.close()
        ref.close()


@pytest.mark.parametrize("heads,kv,ff,kind", [(9, 3, 1536, "q8_0"), (9, 3, 1536, "q4_0"), (12, 4, 1024, "q8_0"), (6, 2, 1024, "q8_0"), (6, 2, 1024, "q4_0")])
def test_no_coarser_beside_channels_that_stand_out(cuda_backend, general, heads, kv, ff, kind):
    """gate and up against 64 bits where one channel of the normed row is 30 000 times the others and its weights are zero: what is left is the grid that the others are cut
    on, 2^-24 of the largest value of their range.  The ranges are those of the general schedule, so the errors are alike over all places of the channel (a tenth for the other
    order of sums)."""
    from zgml_b200 import ProgramIO, abi
    width = 64 * heads
    cfg = LlamaConfig(vocab_size=8, d_model=width, n_layers=1, n_heads=heads, n_kv_heads=kv, d_ff=ff, max_seq_len=8)
    err = {}
    for record in range(width // 32):
        w, k = synthetic_weights(cfg, kind, seed=record, embed_scale=1.0), 32 * record + 5
        w.norm2[0][k] = 3e4
        for name in ("w_gate", "w_up"):
            w.layers[0][name].data.reshape(width, -1)[k] = 0
        for be in (cuda_backend, general):
            s = DeviceLlamaSession(be, cfg, w, 1)
            assert be.program_stats(s.handle)["fused_decode_layers"] == (1 if be is cuda_backend else 0)
            ops = s.lp.program.ops
            at = [i for i, op in enumerate(ops) if op.tag == abi.OP_QMATMUL]          # q, k, v, o, gate, up, down
            bufs = [np.zeros(n, np.float32) for n in s.lp.program.buffer_sizes]
            s.outputs = [ProgramIO(i, b) for i, b in enumerate(bufs)]
            s.execute_at([1], 0)
            x = bufs[ops[at[3] + 1].u.elementwise.dst].astype(np.float64)              # x after attention
            x = x / np.sqrt((x ** 2).mean() + cfg.rms_norm_eps) * w.norm2[0]
            for name, i in (("w_gate", at[4]), ("w_up", at[5])):
                u = w.layers[0][name]
                want = x @ (u.data * np.repeat(u.scales.astype(np.float64), 32)).reshape(width, -1)
                err.setdefault(be, []).append(np.linalg.norm(bufs[ops[i].u.qmatmul.dst] - want) / np.linalg.norm(want))
            s.close()
    mean = {be: np.sqrt(np.mean(np.square(e))) for be, e in err.items()}
    assert mean[cuda_backend] <= 1.1 * mean[general]


def test_op_by_op_steps_report_no_wait(cuda_backend):
    """Profiled steps run op by op, without the kernel: what its error word held when it was allocated is not an error."""
    from zgml_b200 import DeviceBuffer
    from zgml_b200.backend import last_error
    cfg = LlamaConfig(vocab_size=64, d_model=64, n_layers=1, n_heads=1, n_kv_heads=1, d_ff=64, max_seq_len=16)
    old = [DeviceBuffer(cuda_backend, 512, zero=False) for _ in range(8192)]      # small allocations that leave their contents behind
    for b in old:
        b.upload(np.full(128, -1, np.int32))
    for b in old:
        b.free()
    dev = DeviceLlamaSession(cuda_backend, cfg, synthetic_weights(cfg, "q8_0", seed=1), 1)
    assert cuda_backend.program_stats(dev.handle)["fused_decode_layers"] == 1
    cuda_backend.set_profiling(True)
    try:
        dev.step(3)
    finally:
        cuda_backend.set_profiling(False)
    assert "gave up" not in last_error()
    dev.close()


@pytest.mark.parametrize("dh,heads,kv,ff,seq,kind,taken", [
    (64, 9, 3, 1536, 4096, "q8_0", True), (64, 8, 8, 1376, 512, "q8_0", True), (64, 2, 1, 352, 8192, "q8_0", True),
    (64, 8, 8, 1376, 8192, "q8_0", False), (32, 16, 16, 1376, 2048, "q8_0", False), (64, 6, 6, 1024, 4096, "q8_0", False), (64, 12, 4, 1024, 8192, "q4_0", False),       # the cache's share of a CTA
    (64, 2, 1, 352, 8193, "q8_0", False),                                                                                          # beyond what the rule was measured for
    (64, 12, 4, 2048, 64, "q8_0", False), (64, 12, 3, 2496, 64, "q4_0", False)])                                                   # the weights of a CTA
def test_what_the_form_is_taken_for(cuda_backend, dh, heads, kv, ff, seq, kind, taken):
    """Weights and, up to the last position of the cache, keys and values that 16 SMs stream as fast as the general schedule takes."""
    cfg = LlamaConfig(vocab_size=8, d_model=dh * heads, n_layers=1, n_heads=heads, n_kv_heads=kv, d_ff=ff, max_seq_len=seq)
    dev = DeviceLlamaSession(cuda_backend, cfg, synthetic_weights(cfg, kind, seed=1), 1)
    assert cuda_backend.program_stats(dev.handle)["fused_decode_layers"] == int(taken)
    dev.close()


def test_layers_beyond_its_size_keep_the_general_schedule(cuda_backend):
    cfg = LlamaConfig(vocab_size=64, d_model=1024, n_layers=1, n_heads=16, n_kv_heads=4, d_ff=2048, max_seq_len=64)      # 9.5 MB of Q8_0
    dev = DeviceLlamaSession(cuda_backend, cfg, synthetic_weights(cfg, "q8_0", seed=1), 1)
    assert cuda_backend.program_stats(dev.handle)["fused_decode_layers"] == 0
    dev.close()
