"""The plain forms of the one-row product against the general one (which a call takes when it asks for the accumulators):
both do the same arithmetic in the same order, so outputs are bit-equal.  Lengths around the edges of a form: one block,
the last block of a thread's share, 4096 and 8192 where the forms change, and those whose scalar tail has no plain form."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

dev = importlib.import_module("litespark_inference_b200.torchless.device")
K = importlib.import_module("litespark_inference_b200.torchless.kernel")
synthetic = importlib.import_module("litespark_inference_b200.torchless.synthetic")


def _weight(rng, N, n):
    codes = rng.integers(0, 3, (N, n // 4, 4)).astype(np.uint8)
    return dev.DeviceWeight(codes[..., 0] | codes[..., 1] << 2 | codes[..., 2] << 4 | codes[..., 3] << 6, float(rng.uniform(0.5, 2)))


@pytest.mark.parametrize("n", [16, 64, 1008, 2560, 4080, 4096, 4112, 6912, 8176, 8192, 8208, 20, 4100])
@pytest.mark.parametrize("prologue", ["int8", "quant", "norm bf16", "norm fp32", "gated"])
def test_plain_forms_equal_the_general_one(n, prologue):
    rng = np.random.default_rng(n)
    x = dev.DeviceArray.from_numpy((rng.standard_normal(n) * 3).astype(np.float32))
    g = (1.0 + 0.2 * rng.standard_normal(n)).astype(np.float32)
    kw = {"x_f32": x}
    if prologue == "int8":
        kw = {"x_i8": dev.DeviceArray.from_numpy(rng.integers(-127, 128, n).astype(np.int8)),
              "x_scales": dev.DeviceArray.from_numpy(np.float32([0.013]))}
    elif prologue != "quant":
        kw["gamma"] = dev.DeviceArray.from_numpy(g if prologue == "norm fp32" else synthetic.fp32_to_bf16_u16(g))
        if prologue == "gated":
            kw["gate_f32"] = dev.DeviceArray.from_numpy(rng.standard_normal(n).astype(np.float32))
    sizes = {"store": (5000, 16, 40), "add": (4760,), "relu2": (4776, 4776), "silu": (40, 40)}
    for name, epilogue in (("store", K.EPI_STORE), ("add", K.EPI_ADD), ("relu2", K.EPI_RELU2_MUL), ("silu", K.EPI_SILU_MUL)):
        ws = [_weight(rng, N, n) for N in sizes[name]]
        start = [rng.standard_normal(N).astype(np.float32) for N in sizes[name]]
        got = []
        for taps in (False, True):
            outs = [dev.DeviceArray.from_numpy(s) for s in start]
            accs = [dev.DeviceArray((N,), np.int32) for N in sizes[name]] if taps else []
            dev.linear(ws, outs, 1, epilogue=epilogue, acc_outs=accs, **kw)
            got.append([o.numpy() for o in outs])
        for plain, general in zip(*got):
            assert np.array_equal(plain, general, equal_nan=True)
        for w in ws:
            w.free()
