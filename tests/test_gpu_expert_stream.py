"""The expert-grouped products of the MoE layer (several tokens) at the edges of their tiling: rows of an odd number of
64-weight chunks and of lengths that are no multiple of 16, row groups that are not full, experts with more than the
eight rows of a pass, with one row and with none, as many experts as a warp has lanes, both experts for every token."""
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


@pytest.mark.parametrize("hidden,inter,experts,B", [
    (64, 68, 2, 2),            # both experts hold every token; one chunk, a second one of four weights
    (260, 1044, 3, 13),        # 5 and 17 chunks, K % 16 = 4, 26 rows over 3 experts: passes of eight and a remainder
    (512, 2720, 32, 3),        # at most six of 32 experts have rows; 43 chunks: more than one stage, the last one short
    (2560, 6912, 4, 9),        # the model's matrices: many stages, slots reused
    (256, 16 * 150, 8, 70),    # more row groups than CTAs of a pass, 140 rows
])
def test_expert_products_match_oracle(port, hidden, inter, experts, B):
    cfg = hyb.HybridConfig(hidden_size=hidden, num_layers=2, vocab_size=64, num_experts=experts, intermediate_size=inter,
                           nheads=2, headdim=64, d_state=128)
    layer = next(L for L in hyb.random_hybrid(cfg, seed=hidden, norm_jitter=0.1).layers if L.kind == "moe")
    x = np.random.default_rng(B).standard_normal((B, hidden)).astype(np.float32)
    dm = hyb.DeviceMoE(layer, cfg.rms_norm_eps)
    dx = dev.DeviceArray.from_numpy(x)
    sel = dev.DeviceArray((B, 2), np.int32)
    ag, au = dev.DeviceArray((2 * B, inter), np.int32), dev.DeviceArray((2 * B, inter), np.int32)
    ad = dev.DeviceArray((2 * B, hidden), np.int32)
    for a in (ag, au, ad):
        a.fill_bytes(0x7f)                 # a row that nothing wrote differs from every product
    dm.forward(dx, B, sel, None, ag, au, ad)
    got, gsel, gag, gau, gad = dx.numpy(), sel.numpy(), ag.numpy(), au.numpy(), ad.numpy()
    dm.free()
    assert np.abs(gad).max() <= 127 * inter
    exact = 0
    for t in range(0, B, max(1, B // 12)):
        q8, _, routed, _ = ob.moe_route(port, layer, x[t], cfg.rms_norm_eps)
        assert list(gsel[t]) == list(routed)
        for slot, e in enumerate(routed):
            wg, wu = port.acc_int32(q8, layer.gate(e)), port.acc_int32(q8, layer.up(e))
            # an fp32 sum of squares in another order may move single activations by one step of int8: each moves an
            # accumulator by at most 1, and a handful per row is the most seen; identical activations are exact
            assert np.abs(gag[2 * t + slot] - wg).max() <= 4 and np.abs(gau[2 * t + slot] - wu).max() <= 4
            exact += int(np.array_equal(gag[2 * t + slot], wg) and np.array_equal(gau[2 * t + slot], wu))
        want = ob.moe_layer_step(port, layer, x[t], cfg.rms_norm_eps)
        # one of 127 steps of the second quantiser, on an output that sums sqrt(inter) of them: below 5e-3 of its peak
        assert np.abs(got[t] - want).max() <= 5e-3 * np.abs(want - x[t]).max()
    assert exact > 0


def test_many_passes_equal_single_tokens():
    """The model's matrices and enough rows that a CTA's share turns the ring of the down stage (17 slots at K = 6912)
    several times, where every slot has to keep its requesting warp: each row as the one-token kernels compute it, which
    are other code and share its integer sums and roundings, so equal to the bit; and the same again on every run."""
    cfg = hyb.HybridConfig(hidden_size=2560, num_layers=2, vocab_size=64, num_experts=8, intermediate_size=6912, nheads=2,
                           headdim=64, d_state=128)
    layer = next(L for L in hyb.random_hybrid(cfg, seed=8, norm_jitter=0.1).layers if L.kind == "moe")
    dm = hyb.DeviceMoE(layer, cfg.rms_norm_eps)
    B = 64
    x = np.random.default_rng(64).standard_normal((B, 2560)).astype(np.float32)
    runs = []
    for _ in range(6):
        dx = dev.DeviceArray.from_numpy(x)
        dm.forward(dx, B)
        runs.append(dx.numpy())
    assert all(np.array_equal(r, runs[0]) for r in runs)
    for t in range(B):
        one = dev.DeviceArray.from_numpy(x[t:t + 1])
        dm.forward(one, 1)
        assert np.array_equal(one.numpy()[0], runs[0][t]), t
    dm.free()


@pytest.mark.parametrize("hidden,inter", [(320, 200), (64, 4864), (5120, 64)])     # passes of 32 rows; down of 16; gate / up of 16
@pytest.mark.parametrize("B", [41, 48, 57, 64, 65, 81])
def test_passes_of_several_tiles(hidden, inter, B):
    """Two experts, so that each has every token's row: tiles and passes that end anywhere.  Integer sums and the same
    roundings in every form, so each row as the one-token kernels compute it."""
    cfg = hyb.HybridConfig(hidden_size=hidden, num_layers=2, vocab_size=64, num_experts=2, intermediate_size=inter, nheads=2,
                           headdim=64, d_state=128)
    layer = next(L for L in hyb.random_hybrid(cfg, seed=3, norm_jitter=0.1).layers if L.kind == "moe")
    dm = hyb.DeviceMoE(layer, cfg.rms_norm_eps)
    x = np.random.default_rng(B).standard_normal((B, hidden)).astype(np.float32)
    dx = dev.DeviceArray.from_numpy(x)
    dm.forward(dx, B)
    got = dx.numpy()
    for t in range(B):
        one = dev.DeviceArray.from_numpy(x[t:t + 1])
        dm.forward(one, 1)
        assert np.array_equal(one.numpy()[0], got[t]), t
    dm.free()
