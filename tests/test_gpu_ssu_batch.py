"""The Mamba-2 state update of four and more sequences: one head and many, few sequences and more than a hundred."""
import importlib
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "oracle"))
import oracle_blocks as ob  # noqa: E402

hyb = importlib.import_module("litespark_inference_b200.torchless.hybrid")
dev = importlib.import_module("litespark_inference_b200.torchless.device")


@pytest.mark.parametrize("nheads,B", [(1, 4), (4, 5), (20, 40), (80, 4), (13, 150)])
def test_batched_state_update_matches_oracle(port, nheads, B):
    cfg = hyb.HybridConfig(hidden_size=256, num_layers=2, vocab_size=64, num_experts=2, intermediate_size=64, nheads=nheads,
                           headdim=64, d_state=128)
    layer = next(L for L in hyb.random_hybrid(cfg, seed=nheads, norm_jitter=0.1).layers if L.kind == "mamba")
    dmb = hyb.DeviceMamba(layer, cfg.hidden_size, cfg.rms_norm_eps)
    state = dev.DeviceArray((B, dmb.state_floats), np.float32)
    state.fill_bytes(0)
    picked = sorted({0, 1, B // 2, B - 1})
    ost = {b: ob.MambaState(layer) for b in picked}
    rng = np.random.default_rng(B)
    for step in range(5):                  # more steps than the conv ring has slots
        x = rng.standard_normal((B, cfg.hidden_size)).astype(np.float32)
        dx = dev.DeviceArray.from_numpy(x)
        dmb.step(dx, state, dev.DeviceArray.from_numpy(np.full(B, step, np.int32)), B)
        got, st = dx.numpy(), state.numpy()
        for b in picked:
            want = ob.mamba_layer_step(port, layer, ost[b], x[b], cfg.rms_norm_eps)
            # the tolerances of test_gpu_hybrid.py: one of 127 quantiser steps on the output, fp32 sums on the state
            assert np.abs(got[b] - want).max() <= 5e-3 * np.abs(want - x[b]).max(), (step, b)
            ssm = st[b, layer.conv_dim * 4:].reshape(nheads, 64, 128)
            assert np.allclose(ssm, ost[b].ssm, rtol=1e-4, atol=1e-4 * np.abs(ost[b].ssm).max()), (step, b)
    dmb.free()


@pytest.mark.parametrize("B", [8, 9, 16, 33])
def test_a_sequence_does_not_depend_on_its_batch(B):
    """Projections of one row, of eight-row tiles and of the tensor-core GEMM: the same integer sums and the same roundings."""
    cfg = hyb.HybridConfig(hidden_size=256, num_layers=2, vocab_size=64, num_experts=2, intermediate_size=64, nheads=5,
                           headdim=64, d_state=128)
    layer = next(L for L in hyb.random_hybrid(cfg, seed=2, norm_jitter=0.1).layers if L.kind == "mamba")
    dmb = hyb.DeviceMamba(layer, cfg.hidden_size, cfg.rms_norm_eps)
    x = np.random.default_rng(B).standard_normal((B, cfg.hidden_size)).astype(np.float32)

    def step(rows):
        state = dev.DeviceArray((len(rows), dmb.state_floats), np.float32)
        state.fill_bytes(0)
        dx = dev.DeviceArray.from_numpy(rows)
        dmb.step(dx, state, dev.DeviceArray.from_numpy(np.zeros(len(rows), np.int32)), len(rows))
        return dx.numpy(), state.numpy()

    got, states = step(x)
    for b in (0, B // 2, B - 1):
        one, state = step(x[b:b + 1])
        assert np.array_equal(got[b], one[0]) and np.array_equal(states[b], state[0])
    dmb.free()
