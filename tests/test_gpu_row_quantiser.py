"""The row quantiser and the fused prologue of the one-row product: rows of every length at which their split of a row
changes (blocks of 16, the second block per thread from 4096 elements on, 8192), the scalar tail, few and many rows,
bf16 and fp32 norm weights.  The quantiser is bit-equal to the oracle; behind a norm the two kernels are bit-equal to one
another (one order for the sum of squares) and follow the oracle's quantiser from the oracle's norm up to the rounding of
that sum: 16-lane chains there, a 256-lane tree here, each within 1e-6 relative, which moves a scale by as much and an
element by at most one step."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

K = importlib.import_module("litespark_inference_b200.torchless.kernel")
dev = importlib.import_module("litespark_inference_b200.torchless.device")
synthetic = importlib.import_module("litespark_inference_b200.torchless.synthetic")

LENGTHS = [4, 12, 16, 60, 64, 508, 512, 516, 1024, 2560, 4092, 4096, 4100, 5120, 6912, 8188, 8192, 8196]


def _rows(x, gamma, eps):
    T, n = x.shape
    lib = K.load_library()
    dx, q, s = dev.DeviceArray.from_numpy(x), dev.DeviceArray((T, n), np.int8), dev.DeviceArray((T,), np.float32)
    if gamma is None:
        K.check(lib.lspk_quantize_rows(dx.ptr, q.ptr, s.ptr, T, n))
    else:
        dg = dev.DeviceArray.from_numpy(gamma)
        K.check(lib.lspk_rmsnorm_quantize_rows(dx.ptr, dg.ptr, int(gamma.dtype == np.uint16), q.ptr, s.ptr, T, n, eps))
    return q.numpy(), s.numpy()


def _one_row(x, gamma, eps, w):
    """(int8 row, scale, int32 sums) of the one-row product's prologue."""
    n = x.shape[0]
    q, s = dev.DeviceArray((n,), np.int8), dev.DeviceArray((1,), np.float32)
    y, acc = dev.DeviceArray((w.N,), np.float32), dev.DeviceArray((w.N,), np.int32)
    dx, dg = dev.DeviceArray.from_numpy(x), dev.DeviceArray.from_numpy(gamma)
    dev.linear([w], [y], 1, x_f32=dx, gamma=dg, eps=eps, acc_outs=[acc], xq_out=q, xscale_out=s)
    return q.numpy(), s.numpy()[0], acc.numpy()


@pytest.mark.parametrize("n", LENGTHS)
@pytest.mark.parametrize("T,bits", [(1, 16), (3, 32), (150, 16)])
def test_rows_of_every_length(port, n, T, bits):
    rng = np.random.default_rng(n + T)
    x = (rng.standard_normal((T, n)) * np.exp(rng.uniform(-4, 4, (T, 1)))).astype(np.float32)
    x[T // 2, n // 2] *= 30.0
    q, s = _rows(x, None, 0.0)
    wq, ws = np.empty((T, n), np.int8), np.empty(T, np.float32)
    port.quantize_activation_batched(x, wq, ws)
    assert np.array_equal(q, wq) and np.array_equal(s, ws)

    g = (1.0 + 0.2 * rng.standard_normal(n)).astype(np.float32)
    gamma = synthetic.fp32_to_bf16_u16(g) if bits == 16 else g
    q, s = _rows(x, gamma, 1e-5)
    w = dev.DeviceWeight(np.full((16, n // 4), 0xAA, np.uint8), 1.0)          # every weight 1: the sum of the row
    for t in sorted({0, T // 2, T - 1}):
        q1, s1, acc = _one_row(x[t], gamma, 1e-5, w)
        assert np.array_equal(q1, q[t]) and s1 == s[t]
        assert (acc == q[t].astype(np.int64).sum()).all()
    if bits == 16:
        port.rmsnorm_quantize_batched(x, gamma, wq, ws, np.empty((T, n), np.float32), 1e-5)
        assert np.allclose(s, ws, rtol=2e-6, atol=0)
        assert np.abs(q.astype(np.int32) - wq.astype(np.int32)).max() <= 1
    # several rows through a product: the permuted layout and the rows' sums
    y, acc = dev.DeviceArray((T, 16), np.float32), dev.DeviceArray((T, 16), np.int32)
    dx, dg = dev.DeviceArray.from_numpy(x), dev.DeviceArray.from_numpy(gamma)
    dev.linear([w], [y], T, x_f32=dx, gamma=dg, eps=1e-5, acc_outs=[acc])
    assert (acc.numpy() == q.astype(np.int64).sum(axis=1)[:, None]).all()
    w.free()


@pytest.mark.parametrize("n", [60, 2560, 6912])
def test_rows_that_are_not_finite(port, n):
    """An infinity makes the scale infinite and every element 0; elements that are not a number quantise to 0."""
    x = np.random.default_rng(n).standard_normal((4, n)).astype(np.float32)
    x[0, 3], x[1, n // 2], x[1, 5], x[2, :] = np.inf, np.nan, np.nan, 0.0
    q, s = _rows(x, None, 0.0)
    assert np.isinf(s[0]) and not q[0].any()
    clean = x[1].copy()
    clean[[5, n // 2]] = 0.0
    want = np.empty(n, np.int8)
    ws = port.quantize_activation(clean, want)
    assert s[1] == np.float32(ws) and np.array_equal(q[1], want)
    assert not q[2].any() and s[2] == np.float32(np.float32(1e-5) / np.float32(127.0))


@pytest.mark.parametrize("M", [1, 2, 9])
@pytest.mark.parametrize("n", [60, 64, 2560, 2564, 6912, 6916, 8256])
def test_products_of_rows_that_are_not_finite(port, n, M):
    """The same through the products, whose kernels quantise on their own: with and without taps (a form of its own each), with
    and without a norm.  Every row of a call is the same, so one row and several agree.  The elements that are not a number lie
    in a whole block of 16 and in the last, shorter one."""
    rng = np.random.default_rng(n)
    codes = rng.integers(0, 3, (40, n // 4, 4)).astype(np.uint8)
    w = dev.DeviceWeight(codes[..., 0] | codes[..., 1] << 2 | codes[..., 2] << 4 | codes[..., 3] << 6, 1.0)
    plain = codes.reshape(40, n).astype(np.int64) - 1
    g = np.ones(n, np.float32)
    g[[7, n - 2]] = np.nan                       # behind a norm: of the weights, since one in the row makes all of it so
    for bad, norm in ((np.nan, False), (np.inf, False), (np.nan, True)):
        row = rng.standard_normal(n).astype(np.float32)
        if not norm:
            row[[7, n // 2, n - 2]] = bad, -bad, bad
        kw = {"x_f32": dev.DeviceArray.from_numpy(np.tile(row, (M, 1)))}
        if norm:
            kw["gamma"] = dev.DeviceArray.from_numpy(g)
        y, y_plain, acc = dev.DeviceArray((M, 40), np.float32), dev.DeviceArray((M, 40), np.float32), dev.DeviceArray((M, 40), np.int32)
        q, s = dev.DeviceArray((M, n), np.int8), dev.DeviceArray((M,), np.float32)
        dev.linear([w], [y], M, acc_outs=[acc], xq_out=q, xscale_out=s, **kw)
        dev.linear([w], [y_plain], M, **kw)
        clean = row if not norm else (row / np.sqrt((row.astype(np.float64) ** 2).mean() + 1e-5)).astype(np.float32)
        clean = np.where(np.isfinite(clean * g if norm else clean), clean, np.float32(0))
        want = np.zeros(n, np.int8)
        ws = np.float32(np.inf) if bad == np.inf else np.float32(port.quantize_activation(clean, want))
        if bad == np.inf:
            want[:] = 0
        assert np.allclose(s.numpy(), ws, rtol=2e-6, atol=0)
        assert np.abs(q.numpy().astype(int) - want).max() <= (1 if norm else 0) and not q.numpy()[:, ~np.isfinite(g if norm else row)].any()
        sums = q.numpy().astype(np.int64) @ plain.T
        assert np.array_equal(acc.numpy(), sums)
        with np.errstate(invalid="ignore"):
            out = sums.astype(np.float32) * s.numpy()[:, None]
        assert np.array_equal(y.numpy(), out, equal_nan=True) and np.array_equal(y_plain.numpy(), out, equal_nan=True)
    w.free()
