"""The drop-in calls on host pointers: small calls go through a pinned buffer that the GPU reads and writes over the bus,
larger ones through copies.  Both sides of the limit (256 KB each way) against the oracle, in place where the reference
allows it, and from several threads at once."""
import ctypes
import importlib
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

K = importlib.import_module("litespark_inference_b200.torchless.kernel")
LIMIT = 256 * 1024


@pytest.mark.parametrize("T,n", [(1, 1), (1, 2560), (1, 6912), (1, LIMIT // 8), (1, LIMIT // 8 + 1), (9, 6912), (10, 6912), (26, 2560)])
def test_elementwise_calls(port, T, n):
    lib = K.load_library(True)
    rng = np.random.default_rng(T * n)
    g, u = (rng.standard_normal((T, n)).astype(np.float32) for _ in range(2))
    r = np.maximum(g, np.float32(0))
    out = g.copy()
    lib.relu2_mul_fp32_batched_sm100(out, u, out, T, n)          # in place
    assert np.array_equal(out, r * r * u)
    a = g.ravel().copy()
    lib.add_inplace_fp32_sm100(a, u.ravel(), a.size)
    assert np.array_equal(a, g.ravel() + u.ravel())


@pytest.mark.parametrize("T,n", [(1, 4), (1, 2560), (1, 8192), (9, 6912), (10, 6912), (25, 2560), (26, 2560)])
def test_rows_and_products(port, T, n):
    lib = K.load_library(True)
    rng = np.random.default_rng(T + n)
    x = rng.standard_normal((T, n)).astype(np.float32)
    q, s = np.empty((T, n), np.int8), np.empty(T, np.float32)
    lib.quantize_activation_batched_sm100(x, q, s, T, n)
    wq, ws = np.empty_like(q), np.empty_like(s)
    port.quantize_activation_batched(x, wq, ws)
    assert np.array_equal(q, wq) and np.array_equal(s, ws)
    for N in (16, LIMIT // 4 // T, LIMIT // 4 // T + 1):
        if N * n > 1 << 26:
            continue
        packed = rng.integers(0, 3, (N, n // 4), dtype=np.uint8) * np.uint8(0x55)      # four equal weights a byte
        w = (packed & 3).astype(np.float64) - 1
        y = np.empty((T, N), np.float32)
        lib.matmul_lut_sm100_mT(q, s, packed, np.float32(0.5), y, T, N, n)
        dots = q.astype(np.float64).reshape(T, n // 4, 4).sum(axis=2) @ w.T            # exact: integers below 2^53
        assert np.array_equal(y, dots.astype(np.float32) * (s * np.float32(0.5))[:, None])


@pytest.mark.parametrize("T,n", [(1, 16), (1, 2560), (1, 2562), (1, 8192), (1, 12288), (9, 6912), (10, 6912), (23, 2560), (24, 2560), (26, 2560),
                                 (24, 2562), (30, 2048), (512, 64), (4096, 4), (4097, 4)])
def test_norms_of_changing_weights(port, T, n):
    """Calls of one shape one behind the other, each with norm weights (and rows) of its own: all pass through the same buffer.
    The sum of squares is summed in another order than the oracle's: 2e-6 relative, and an element may round the other way."""
    lib = K.load_library(True)
    rng = np.random.default_rng(T + n)
    o, q, s = np.empty((T, n), np.float32), np.empty((T, n), np.int8), np.empty(T, np.float32)
    wq, ws, tmp = np.empty_like(q), np.empty_like(s), np.empty_like(o)
    for i in range(12):
        x = rng.standard_normal((T, n)).astype(np.float32)
        g32 = ((1 + i) * rng.uniform(0.5, 1.5, n)).astype(np.float32)
        g16 = (g32.view(np.uint32) >> 16).astype(np.uint16)
        lib.rmsnorm_quantize_bf16gamma_batched_sm100(x, g16, q, s, tmp, T, n, 1e-5)
        port.rmsnorm_quantize_batched(x, g16, wq, ws, tmp, 1e-5)
        assert np.allclose(s, ws, rtol=2e-6, atol=0) and np.abs(q.astype(np.int32) - wq).max() <= 1
        for norm, gamma in ((lib.rmsnorm_bf16gamma_fp32_batched_sm100, g16), (lib.rmsnorm_fp32gamma_fp32_batched_sm100, g32)):
            norm(x, gamma, o, T, n, 1e-5)
            g = g32 if gamma is g32 else (g16.astype(np.uint32) << 16).view(np.float32)
            wo = (x / np.sqrt((x.astype(np.float64) ** 2).mean(axis=1, keepdims=True) + 1e-5) * g).astype(np.float32)
            assert np.allclose(o, wo, rtol=2e-6, atol=0)


@pytest.mark.parametrize("T,n", [(1, 2560), (40, 2560)])
def test_null_outputs(T, n):
    """On either side of the limit: a null fp32 row or null scales are recorded as a failure, null int8 rows are left out."""
    lib = ctypes.CDLL(str(K.library_path()))          # plain pointers, past the array checks of the wrappers
    lib.lspk_last_error.restype = ctypes.c_char_p
    x, gamma = np.random.default_rng(n).standard_normal((T, n)).astype(np.float32), np.full(n, 0x3f80, np.uint16)
    q, s, s_alone = np.empty((T, n), np.int8), np.empty(T, np.float32), np.zeros(T, np.float32)
    at = lambda a: None if a is None else ctypes.c_void_p(a.ctypes.data)  # noqa: E731
    eps, rows, width = ctypes.c_float(1e-5), ctypes.c_int(T), ctypes.c_int(n)
    quantise = lambda o, sc: lib.quantize_activation_batched_sm100(at(x), at(o), at(sc), rows, width)  # noqa: E731
    norm_quantise = lambda o, sc: lib.rmsnorm_quantize_bf16gamma_batched_sm100(  # noqa: E731
        at(x), at(gamma), at(o), at(sc), None, rows, width, eps)
    failing = [lambda: lib.rmsnorm_bf16gamma_fp32_batched_sm100(at(x), at(gamma), None, rows, width, eps),
               lambda: lib.rmsnorm_fp32gamma_fp32_batched_sm100(at(x), at(x), None, rows, width, eps),
               lambda: quantise(q, None), lambda: norm_quantise(q, None),
               lambda: lib.relu2_mul_fp32_batched_sm100(at(x), at(x), None, rows, width)]
    for call in failing:
        lib.lspk_clear_error()
        call()
        assert lib.lspk_error_count() == 1 and any(m in lib.lspk_last_error() for m in (b"null output", b"bad arguments"))
    lib.lspk_clear_error()
    for call in (quantise, norm_quantise):
        call(q, s)
        call(None, s_alone)
        assert lib.lspk_error_count() == 0 and np.array_equal(s, s_alone)


def test_calls_from_several_threads():
    lib = K.load_library(True)
    rng = np.random.default_rng(0)
    data = [(rng.standard_normal(n).astype(np.float32), rng.standard_normal(n).astype(np.float32)) for n in (5, 2560, 6912, 40000)]
    bad = []

    def work(a, b):
        for _ in range(50):
            got = a.copy()
            lib.add_inplace_fp32_sm100(got, b, got.size)
            if not np.array_equal(got, a + b):
                bad.append(a.size)

    threads = [threading.Thread(target=work, args=d) for d in data]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
