"""LINEAR of many rows over f32 weights (operands cut into three bfloat16 parts on the tensor cores) against float64: edges of the 128 x 128 tiles and of
the 64-k steps, one and several shares of K, strided rows, bias, activation on part of the columns, gated pairs, magnitudes that differ between rows and
within a row, sums near the largest float, more rows than a grid has in y, and rows that hold an infinity or a NaN.

Tolerance: three parts hold every operand whole, the products left out are below 2^-25 of one product, a 64-k step adds four truncated f32 sums and up to
100 steps add in f32: 3e-6 of sqrt(K) |x| |w| is over three times what that makes; the plain f32 sum shows about 1e-6."""
import numpy as np
import pytest

from test_gpu_recops import run, sigmoid, weights

pytestmark = pytest.mark.gpu


def check(got, x, W, want):
    bound = 3e-6 * np.linalg.norm(x.astype(np.float64), axis=1)[:, None] * np.linalg.norm(W.astype(np.float64), axis=1)[None]
    assert (np.abs(got - want) <= bound).all()


@pytest.mark.parametrize("M,N,K", [(9, 32, 64), (16, 33, 68), (127, 129, 252), (128, 128, 128), (129, 257, 324), (200, 64, 4096), (300, 1000, 772), (17, 2050, 1536)])
def test_against_float64(cuda_backend, M, N, K):
    from zgml_b200 import DeviceOp, ExternBuffer, abi
    r = np.random.default_rng(M + N + K)
    W = (r.standard_normal((N, K)) * 10.0 ** r.integers(-12, 12, (N, 1))).astype(np.float32)
    x = (r.standard_normal((M, K)) * 10.0 ** r.integers(-9, 9, (M, 1))).astype(np.float32)
    buf, (ow,) = weights(cuda_backend, W)
    wide = np.zeros((M, K + 4), np.float32)
    wide[:, :K] = x
    op = DeviceOp.linear(0, 1, 2, ow, M, N, K, abi.W_F32, src_rs=K + 4, dst_rs=N + 3)
    got = run(cuda_backend, [op], [M * (N + 3), wide.size, buf.elems], [(1, wide)], 0, (M, N + 3), [ExternBuffer(2, buf)])[:, :N]
    check(got, x, W, x.astype(np.float64) @ W.astype(np.float64).T)
    buf.free()


def test_bias_activation_range_and_pairs(cuda_backend):
    from zgml_b200 import DeviceOp, ExternBuffer, abi
    r = np.random.default_rng(1)
    M, N, K = 70, 150, 200
    W, b, x = (r.standard_normal((2 * N, K)) / 14).astype(np.float32), r.standard_normal(N).astype(np.float32), r.standard_normal((M, K)).astype(np.float32)
    buf, (ow, ob) = weights(cuda_backend, W, b)
    z = x.astype(np.float64) @ W.astype(np.float64).T
    ext, sizes = [ExternBuffer(2, buf)], [M * N, x.size, buf.elems]
    got = run(cuda_backend, [DeviceOp.linear(0, 1, 2, ow, M, N, K, abi.W_F32, bias=2, bias_off=ob, act="silu", act_cols=(30, 101))], sizes, [(1, x)], 0, (M, N), ext)
    want = z[:, :N] + b
    want[:, 30:101] *= sigmoid(want[:, 30:101])
    assert np.abs(got - want).max() < 1e-5
    got = run(cuda_backend, [DeviceOp.linear(0, 1, 2, ow, M, N, K, abi.W_F32, act="relu2", pairs=True)], sizes, [(1, x)], 0, (M, N), ext)
    assert np.abs(got - np.maximum(z[:, 0::2], 0) ** 2 * z[:, 1::2]).max() < 3e-5 * np.abs(z).max()
    buf.free()


def test_non_finite_rows(cuda_backend):
    """An infinity times weights of both signs is what the plain sum makes of it; the other rows and columns are as they were."""
    from zgml_b200 import DeviceOp, ExternBuffer, abi
    r = np.random.default_rng(2)
    M, N, K = 40, 64, 128
    W, x = r.standard_normal((N, K)).astype(np.float32), r.standard_normal((M, K)).astype(np.float32)
    x[3, 70], x[17, 5], W[9, 9] = np.inf, np.nan, -np.inf
    buf, (ow,) = weights(cuda_backend, W)
    got = run(cuda_backend, [DeviceOp.linear(0, 1, 2, ow, M, N, K, abi.W_F32)], [M * N, x.size, buf.elems], [(1, x)], 0, (M, N), [ExternBuffer(2, buf)])
    with np.errstate(invalid="ignore"):
        want = x.astype(np.float64) @ W.astype(np.float64).T
    fin = np.isfinite(want)
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(got[~fin & ~np.isnan(want)], want[~fin & ~np.isnan(want)].astype(np.float32))
    assert np.abs(got[fin] - want[fin]).max() < 1e-4
    buf.free()


def waits_given_up(be):
    from zgml_b200 import DeviceOp, DeviceProgram
    h = be.compile_program(DeviceProgram([DeviceOp.rmsnorm(1, 0, 1, 32, 1e-5)], [32, 32], [], []))
    n = be.program_stats(h)["dense_gemm_timeouts"]
    be.free_program(h)
    return n


def linear(be, x, W, **kwargs):
    from zgml_b200 import DeviceOp, ExternBuffer, abi
    (M, K), N = x.shape, len(W)
    buf, (ow,) = weights(be, W)
    got = run(be, [DeviceOp.linear(0, 1, 2, ow, M, N, K, abi.W_F32, **kwargs)], [M * N, x.size, buf.elems], [(1, x)], 0, (M, N), [ExternBuffer(2, buf)])
    buf.free()
    return got


def test_one_hot_weights_return_the_inputs(cuda_backend):
    """Every output is one input, whatever else its row holds: magnitudes from 2^-60 to 2^60 in each row, all 24 bits."""
    r = np.random.default_rng(4)
    M, N, K = 140, 132, 200
    x = (r.standard_normal((M, K)) * 2.0 ** r.integers(-60, 61, (M, K))).astype(np.float32)
    pick = r.integers(0, K, N)
    W = np.zeros((N, K), np.float32)
    W[np.arange(N), pick] = 1.0
    assert np.array_equal(linear(cuda_backend, x, W), x[:, pick])


@pytest.mark.parametrize("where", ["source", "weights"])
def test_large_elements_that_meet_zeros(cuda_backend, where):
    """2^20 to 2^40 beside values around 1, against zeros: the bound is that of the sum without them."""
    r = np.random.default_rng(6)
    M, N, K = 130, 140, 320
    x, W = r.standard_normal((M, K)).astype(np.float32), r.standard_normal((N, K)).astype(np.float32)
    a, b = (x, W) if where == "source" else (W, x)
    rest = np.arange(K) % 16 != 5
    b[:, ~rest] = 0.0
    a[:, ~rest] = 2.0 ** r.integers(20, 41, (len(a), K // 16))
    check(linear(cuda_backend, x, W), x[:, rest], W[:, rest], x.astype(np.float64) @ W.astype(np.float64).T)


@pytest.mark.parametrize("big,small", [(1e33, 1e-3), (1e38, 1e-30), (3e38, 1e-3), (1e-30, 1e28)])
@pytest.mark.parametrize("where", ["source", "weights"])
def test_finite_sums_of_extreme_operands(cuda_backend, big, small, where):
    r = np.random.default_rng(7)
    M, N, K = 20, 130, 192
    x, W = r.uniform(-1, 1, (M, K)), r.uniform(-1, 1, (N, K))
    x, W = (x * (big if where == "source" else small)).astype(np.float32), (W * (small if where == "source" else big)).astype(np.float32)
    want = x.astype(np.float64) @ W.astype(np.float64).T
    assert np.abs(want).max() < 1e37
    check(linear(cuda_backend, x, W), x, W, want)


@pytest.mark.parametrize("M,N,K", [(65535 + 129, 32, 64), (70000, 40, 256)])
def test_more_rows_than_a_grid_has_in_y(cuda_backend, M, N, K):
    r = np.random.default_rng(8)
    x, W = r.standard_normal((M, K)).astype(np.float32), r.standard_normal((N, K)).astype(np.float32)
    check(linear(cuda_backend, x, W), x, W, x.astype(np.float64) @ W.astype(np.float64).T)


def test_no_wait_ran_out(cuda_backend):
    """Statistic 5 of a program counts the waits that its tensor-core kernels gave up on: none, after everything above."""
    assert waits_given_up(cuda_backend) == 0
