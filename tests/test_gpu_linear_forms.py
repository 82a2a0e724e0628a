"""The plain forms of the products against the general one (which a call takes when it asks for the accumulators): both do the
same arithmetic in the same order, so outputs are bit-equal.  Lengths around the edges of a form: one block, the last block
of a thread's share, 4096 and 8192 where the forms change, and those whose scalar tail has no plain form.  Sizes on either
side of the grid: a CTA per row group (forms without the loop), and more row groups than CTAs by the number of SMs."""
import ctypes
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

dev = importlib.import_module("litespark_inference_b200.torchless.device")
K = importlib.import_module("litespark_inference_b200.torchless.kernel")
synthetic = importlib.import_module("litespark_inference_b200.torchless.synthetic")


_TRITS = np.array([a | b << 2 | c << 4 | d << 6 for a in range(3) for b in range(3) for c in range(3) for d in range(3)], np.uint8)


def _weight(rng, N, n):
    return dev.DeviceWeight(_TRITS[rng.integers(0, 81, (N, n // 4), dtype=np.uint8)], float(rng.uniform(0.5, 2)))


def _dots(q, w):
    """Products of int8 rows and a weight's trits; below 2^24, so exact in fp32 in any order."""
    packed = w.download()
    trits = np.stack([(packed >> s & 3) for s in (0, 2, 4, 6)], axis=2).reshape(w.N, w.K).astype(np.float32) - 1
    return q.astype(np.float32) @ trits.T


@pytest.mark.parametrize("n", [16, 64, 1008, 2560, 4080, 4096, 4112, 6912, 8176, 8192, 8208, 20, 4100])
@pytest.mark.parametrize("prologue", ["int8", "quant", "norm bf16", "norm fp32", "gated"])
def test_plain_forms_equal_the_general_one(port, n, prologue):
    rng = np.random.default_rng(n)
    x = dev.DeviceArray.from_numpy((rng.standard_normal(n) * 3).astype(np.float32))
    g = (1.0 + 0.2 * rng.standard_normal(n)).astype(np.float32)
    kw = {"x_f32": x}
    q, s = np.empty(n, np.int8), np.float32(0.013)
    if prologue == "int8":
        q[:] = rng.integers(-127, 128, n)
        kw = {"x_i8": dev.DeviceArray.from_numpy(q), "x_scales": dev.DeviceArray.from_numpy(np.float32([s]))}
    elif prologue == "quant":
        s = np.float32(port.quantize_activation(x.numpy(), q))
    elif prologue != "quant":
        kw["gamma"] = dev.DeviceArray.from_numpy(g if prologue == "norm fp32" else synthetic.fp32_to_bf16_u16(g))
        if prologue == "gated":
            kw["gate_f32"] = dev.DeviceArray.from_numpy(rng.standard_normal(n).astype(np.float32))
    sms = K.load_library(True).lspk_sm_count()       # at most three CTAs per SM take a row group of 16 each, of a pair two
    for sizes, epilogue in (((5000, 16, 40), K.EPI_STORE), ((48 * sms + 8, 16, 40), K.EPI_STORE), ((4760,), K.EPI_ADD),
                            ((48 * sms + 24,), K.EPI_ADD), ((32 * sms + 24,) * 2, K.EPI_RELU2_MUL), ((40, 40), K.EPI_RELU2_MUL),
                            ((40, 40), K.EPI_SILU_MUL)):
        ws = [_weight(rng, N, n) for N in sizes]
        start = [rng.standard_normal(N).astype(np.float32) for N in sizes]
        got = []
        for taps in (False, True):
            outs = [dev.DeviceArray.from_numpy(s) for s in start]
            accs = [dev.DeviceArray((N,), np.int32) for N in sizes] if taps else []
            dev.linear(ws, outs, 1, epilogue=epilogue, acc_outs=accs, **kw)
            got.append([o.numpy() for o in outs])
        for plain, general in zip(*got):
            assert np.array_equal(plain, general, equal_nan=True)
        if prologue in ("int8", "quant") and epilogue in (K.EPI_STORE, K.EPI_ADD):      # the same roundings in the same order
            for y, w, v in zip(got[0], ws, start):
                want = _dots(q, w) * (s * np.float32(w.scale))
                assert np.array_equal(y, want if epilogue == K.EPI_STORE else v + want)
        for w in ws:
            w.free()


@pytest.mark.parametrize("M", [2, 8, 9, 40, 130])
@pytest.mark.parametrize("n", [16, 64, 2560, 4096, 4112, 6912, 8192, 4100])
def test_many_rows_plain_and_general_forms(n, M):
    """Rows normalised and quantised on the way into a product, without accumulators (plain forms of the row quantiser and
    of the product) and with them, and as int8 rows from the quantiser's natural order: one result, bit for bit, that of
    the int8 rows."""
    rng = np.random.default_rng(n + M)
    x = dev.DeviceArray.from_numpy((rng.standard_normal((M, n)) * 3).astype(np.float32))
    gamma = dev.DeviceArray.from_numpy(synthetic.fp32_to_bf16_u16((1.0 + 0.2 * rng.standard_normal(n)).astype(np.float32)))
    q, s = dev.DeviceArray((M, n), np.int8), dev.DeviceArray((M,), np.float32)
    K.check(K.load_library().lspk_rmsnorm_quantize_rows(x.ptr, gamma.ptr, 1, q.ptr, s.ptr, M, n, 1e-5))
    many = 32 * K.load_library(True).lspk_sm_count() + 24       # more row groups than the eight-row kernel has CTAs
    wide = [((many, 16, 40), K.EPI_STORE), ((many,), K.EPI_ADD), ((many, many), K.EPI_RELU2_MUL)] if M <= 9 else []
    for sizes, epilogue in [((200, 16, 40), K.EPI_STORE), ((200,), K.EPI_ADD), ((200, 200), K.EPI_RELU2_MUL),
                            ((40, 40), K.EPI_SILU_MUL)] + wide:
        ws = [_weight(rng, N, n) for N in sizes]
        start = [rng.standard_normal((M, N)).astype(np.float32) for N in sizes]
        got = []
        for rows, taps in (("fp32", False), ("fp32", True), ("int8", False), ("int8", True)):
            outs = [dev.DeviceArray.from_numpy(v) for v in start]
            accs = [dev.DeviceArray((M, N), np.int32) for N in sizes] if taps else []
            kw = {"x_f32": x, "gamma": gamma} if rows == "fp32" else {"x_i8": q, "x_scales": s}
            dev.linear(ws, outs, M, epilogue=epilogue, acc_outs=accs, **kw)
            got.append([o.numpy() for o in outs])
        for other in got[1:]:
            for a, b in zip(got[0], other):
                assert np.array_equal(a, b, equal_nan=True)
        if epilogue == K.EPI_STORE:
            for y, w in zip(got[0], ws):
                assert np.array_equal(y, _dots(q.numpy(), w) * (s.numpy() * np.float32(w.scale))[:, None])
        for w in ws:
            w.free()


@pytest.mark.parametrize("n", [64, 2560, 4096, 4112, 6912, 8192, 8208, 12288])
def test_a_row_launch_is_resident_at_once(n):
    """One row: more than two CTAs per SM only where the registers of the chosen form let an SM hold them."""
    lib, sms = K.load_library(True), K.load_library(True).lspk_sm_count()
    x, q, s = dev.DeviceArray((n,), np.float32), dev.DeviceArray((n,), np.int8), dev.DeviceArray((1,), np.float32)
    g = dev.DeviceArray((n,), np.uint16)
    for N in (16, 32 * sms, 32 * sms + 16, 48 * sms, 48 * sms + 16, 80 * sms):
        w = dev.DeviceWeight(np.full((N, n // 4), 0x55, np.uint8), 1.0)
        y, acc = dev.DeviceArray((N,), np.float32), dev.DeviceArray((N,), np.int32)
        for prologue in (K.PRO_INT8, K.PRO_QUANT, K.PRO_RMSNORM_QUANT, K.PRO_GATED_RMSNORM_QUANT):
            for pair, tap in ((False, False), (False, True), (True, False)):
                a, ctas, resident = K.LinearArgs(), ctypes.c_int(), ctypes.c_int()
                a.n_mats, a.M, a.prologue, a.epilogue, a.gamma_is_bf16 = 1 + pair, 1, prologue, K.EPI_SILU_MUL * pair, 1
                a.x_f32, a.x_i8, a.x_scales, a.gamma, a.gate_f32 = x.ptr, q.ptr, s.ptr, g.ptr, x.ptr
                a.w[0], a.w[1], a.out[0], a.acc_out[0] = w.handle, w.handle if pair else None, y.ptr, acc.ptr if tap else None
                K.check(lib.lspk_debug_row_launch(ctypes.byref(a), ctypes.byref(ctas), ctypes.byref(resident)))
                most = max(2, resident.value) * sms
                assert resident.value >= 1 and 1 <= ctas.value <= most, (N, prologue, pair, tap)
                assert ctas.value == N // 16 or ctas.value >= 2 * sms
        w.free()
