"""What lspk_linear refuses, at row counts of each of its kernels (the one-row kernel, the eight-row tiles, the tensor-memory
GEMM): a call without one of its operands is an argument error and launches nothing."""
import ctypes
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

dev = importlib.import_module("litespark_inference_b200.torchless.device")
K = importlib.import_module("litespark_inference_b200.torchless.kernel")
pack = importlib.import_module("litespark_inference_b200.torchless.pack")

LSPK_ERR_ARG = 1


@pytest.mark.parametrize("M", [1, 8, 9, 31, 32, 200])
def test_missing_operands_are_refused(M):
    N, Kd = 128, 256
    rng = np.random.default_rng(M)
    w = dev.DeviceWeight(pack.pack_ternary_4_per_byte(rng.integers(-1, 2, (N, Kd), dtype=np.int8)), 1.0)
    other = dev.DeviceWeight(pack.pack_ternary_4_per_byte(rng.integers(-1, 2, (N, Kd // 2), dtype=np.int8)), 1.0)
    taller = dev.DeviceWeight(pack.pack_ternary_4_per_byte(rng.integers(-1, 2, (2 * N, Kd), dtype=np.int8)), 1.0)
    xf = dev.DeviceArray.from_numpy(rng.standard_normal((M, Kd)).astype(np.float32))
    xq = dev.DeviceArray.from_numpy(rng.integers(-127, 128, (M, Kd), dtype=np.int8))
    xs = dev.DeviceArray.from_numpy(np.ones(M, np.float32))
    g = dev.DeviceArray.from_numpy(np.full(Kd, 0x3f80, np.uint16))
    y = dev.DeviceArray.from_numpy(np.full((M, N), 7.0, np.float32))
    lib = K.load_library()

    def call(**kw):
        a = K.LinearArgs()
        a.w[0], a.out[0], a.n_mats, a.M, a.eps, a.gamma_is_bf16 = w.handle, y.ptr, 1, M, 1e-5, 1
        for name, value in kw.items():
            if name in ("w", "out"):
                for i, v in enumerate(value):
                    getattr(a, name)[i] = v
            else:
                setattr(a, name, value)
        return lib.lspk_linear(ctypes.byref(a))

    int8, norm = dict(prologue=K.PRO_INT8, x_i8=xq.ptr), dict(prologue=K.PRO_RMSNORM_QUANT, x_f32=xf.ptr)
    refused = [
        dict(int8), dict(prologue=K.PRO_INT8, x_scales=xs.ptr), dict(norm), dict(prologue=K.PRO_RMSNORM_QUANT, gamma=g.ptr),
        dict(prologue=K.PRO_QUANT), dict(prologue=3, x_f32=xf.ptr, gamma=g.ptr), dict(prologue=5, x_f32=xf.ptr),
        dict(int8, x_scales=xs.ptr, epilogue=9), dict(int8, x_scales=xs.ptr, n_mats=0), dict(int8, x_scales=xs.ptr, n_mats=4),
        dict(int8, x_scales=xs.ptr, w=[None]), dict(int8, x_scales=xs.ptr, out=[None]),
        dict(int8, x_scales=xs.ptr, n_mats=2, w=[w.handle, other.handle], out=[y.ptr, y.ptr]),
        dict(int8, x_scales=xs.ptr, n_mats=2, w=[w.handle, w.handle], out=[y.ptr, None]),
        dict(int8, x_scales=xs.ptr, epilogue=K.EPI_RELU2_MUL),
        dict(int8, x_scales=xs.ptr, epilogue=K.EPI_RELU2_MUL, n_mats=2, w=[w.handle, taller.handle]),
    ]
    for kw in refused:
        assert call(**kw) == LSPK_ERR_ARG, kw
    assert (y.numpy() == 7.0).all()
    assert call(**int8, x_scales=xs.ptr) == 0 and call(**norm, gamma=g.ptr) == 0
    K.check(lib.lspk_sync())
