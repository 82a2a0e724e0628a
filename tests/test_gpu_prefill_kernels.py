"""The many-row kernels of the prefill at the edges of their tiles and plans."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

dev = importlib.import_module("litespark_inference_b200.torchless.device")
K = importlib.import_module("litespark_inference_b200.torchless.kernel")
rt = importlib.import_module("litespark_inference_b200.torchless.runtime")
synthetic = importlib.import_module("litespark_inference_b200.torchless.synthetic")
pack = importlib.import_module("litespark_inference_b200.torchless.pack")


@pytest.mark.parametrize("epilogue", [K.EPI_STORE, K.EPI_ADD, K.EPI_RELU2_MUL])
# rows around the token tiles (32, 64, 96, 128); features off the 128-row tile; K off the 256-wide block, K of a single
# block, K long enough for every K split, and grids of several tiles per SM
@pytest.mark.parametrize("M,N,Kd", [(9, 128, 64), (31, 300, 320), (33, 130, 2560), (65, 640, 1024), (97, 257, 448),
                                    (129, 384, 6912), (300, 2560, 512), (700, 1153, 260)])
def test_gemm_tiles_bit_exact(M, N, Kd, epilogue):
    rng = np.random.default_rng(M + N + Kd)
    pair = epilogue == K.EPI_RELU2_MUL
    ws = [np.float32(0.75), np.float32(1.25)][:2 if pair else 1]
    w = [rng.integers(-1, 2, (N, Kd), dtype=np.int8) for _ in ws]
    xq = rng.integers(-127, 128, (M, Kd), dtype=np.int8)
    xs = rng.uniform(0.01, 0.02, M).astype(np.float32)
    res = rng.standard_normal((M, N)).astype(np.float32)
    acc = [xq.astype(np.int32) @ a.T.astype(np.int32) for a in w]
    y = [a.astype(np.float32) * (xs * s)[:, None] for a, s in zip(acc, ws)]
    want = y[0] if epilogue == K.EPI_STORE else res + y[0] if epilogue == K.EPI_ADD else np.maximum(y[0], 0) ** 2 * y[1]
    W = [dev.DeviceWeight(pack.pack_ternary_4_per_byte(a), float(s)) for a, s in zip(w, ws)]
    out = dev.DeviceArray.from_numpy(res)
    taps = [dev.DeviceArray((M, N), np.int32) for _ in W]
    lib = K.load_library()
    try:
        K.check(lib.lspk_linear_force_path(2))
        dev.linear(W, [out, None][:len(W)], M, x_i8=dev.DeviceArray.from_numpy(xq), x_scales=dev.DeviceArray.from_numpy(xs),
                   epilogue=epilogue, acc_outs=taps)
        K.check(lib.lspk_tc_check_error())
    finally:
        lib.lspk_linear_force_path(0)
    for t, a in zip(taps, acc):
        assert np.array_equal(t.numpy(), a)
    assert np.array_equal(out.numpy(), want)      # the same roundings in the same order


# Every (columns, split) that the plan takes for the products of a 2560 / 6912 layer between 9 and 1531 rows on 148 SMs, named
# beside it, and the splits of a pair that small matrices take: the plain form of each, which a call without accumulators
# takes, against the general one and the exact sums (below 2^24, so fp32 holds them in any order of summation).
@pytest.mark.parametrize("pair,sizes,Kd,M", [
    (False, (2560, 640, 640), 2560, 9),       # 32 x 4
    (False, (2560, 640, 640), 2560, 65),      # 64 x 4
    (False, (2560, 640, 640), 2560, 129),     # 64 x 2
    (False, (2560, 640, 640), 2560, 257),     # 32 x 1
    (False, (2560, 640, 640), 2560, 289),     # 96 x 1
    (False, (2560, 640, 640), 2560, 385),     # 64 x 1
    (False, (2560,), 6912, 193),              # 32 x 2
    (False, (2560,), 6912, 225),              # 96 x 2
    (False, (2560,), 6912, 289),              # 64 x 2
    (False, (2560,), 6912, 673),              # 128 x 1
    (False, (2560,), 6912, 1531),             # 128 x 1, the last tile in part
    (True, (6912, 6912), 2560, 9),           # 32 x 2
    (True, (6912, 6912), 2560, 33),          # 64 x 2
    (True, (6912, 6912), 2560, 65),          # 64 x 1
    (True, (6912, 6912), 2560, 129),         # 96 x 1
    (True, (6912, 6912), 2560, 193),         # 128 x 1
    (True, (6912, 6912), 2560, 512),         # 128 x 1
    (True, (1000, 1000), 2560, 100),         # 32 x 4
    (True, (1000, 1000), 2560, 129),         # 64 x 4
])
def test_gemm_plans_without_taps(pair, sizes, Kd, M):
    rng = np.random.default_rng(M + Kd)
    xq, xs = rng.integers(-127, 128, (M, Kd), dtype=np.int8), rng.uniform(0.01, 0.02, M).astype(np.float32)
    scales = [np.float32(0.75), np.float32(1.25), np.float32(0.5)][:len(sizes)]
    w = [rng.integers(-1, 2, (N, Kd), dtype=np.int8) for N in sizes]
    y = [(xq.astype(np.float32) @ a.T.astype(np.float32)) * (xs * s)[:, None] for a, s in zip(w, scales)]
    W = [dev.DeviceWeight(pack.pack_ternary_4_per_byte(a), float(s)) for a, s in zip(w, scales)]
    dx, ds = dev.DeviceArray.from_numpy(xq), dev.DeviceArray.from_numpy(xs)
    start = [rng.standard_normal((M, N)).astype(np.float32) for N in sizes]
    lib = K.load_library()
    for epilogue in (K.EPI_RELU2_MUL, K.EPI_SILU_MUL) if pair else (K.EPI_STORE, K.EPI_ADD):
        got = []
        for taps in (False, True):
            outs = [dev.DeviceArray.from_numpy(v) for v in (start[:1] if pair else start)]
            accs = [dev.DeviceArray((M, N), np.int32) for N in sizes] if taps else []
            try:
                K.check(lib.lspk_linear_force_path(2))
                dev.linear(W, [*outs, None][:len(W)], M, x_i8=dx, x_scales=ds, epilogue=epilogue, acc_outs=accs)
                K.check(lib.lspk_tc_check_error())
            finally:
                lib.lspk_linear_force_path(0)
            got.append([o.numpy() for o in outs])
        for plain, general in zip(*got):
            assert np.array_equal(plain, general)
        if epilogue == K.EPI_SILU_MUL:      # the exponential's error against the processor's: a few units in the last place
            with np.errstate(over="ignore"):
                assert np.allclose(got[0][0], y[0] / (1 + np.exp(-y[0])) * y[1], rtol=1e-5, atol=1e-6)
        elif pair:
            assert np.array_equal(got[0][0], np.maximum(y[0], 0) ** 2 * y[1])
        else:
            for a, b, v in zip(got[0], y, start):
                assert np.array_equal(a, b if epilogue == K.EPI_STORE else v + b)
    for x in W:
        x.free()


@pytest.mark.parametrize("M", [8, 9, 16, 17, 24])
@pytest.mark.parametrize("Kd", [4, 68, 2560, 4100])          # rows of one word, off the 16-element block, of several trips
def test_int8_rows_on_either_side_of_the_choice_of_a_kernel(M, Kd):
    rng = np.random.default_rng(M + Kd)
    N = 130
    w, xq = rng.integers(-1, 2, (N, Kd), dtype=np.int8), rng.integers(-127, 128, (M, Kd), dtype=np.int8)
    xs = rng.uniform(0.01, 0.02, M).astype(np.float32)
    W = dev.DeviceWeight(pack.pack_ternary_4_per_byte(w), 0.75)
    out, acc = dev.DeviceArray((M, N), np.float32), dev.DeviceArray((M, N), np.int32)
    dev.linear([W], [out], M, x_i8=dev.DeviceArray.from_numpy(xq), x_scales=dev.DeviceArray.from_numpy(xs), acc_outs=[acc])
    want = xq.astype(np.int32) @ w.T.astype(np.int32)
    assert np.array_equal(acc.numpy(), want)
    assert np.array_equal(out.numpy(), want.astype(np.float32) * (xs * np.float32(0.75))[:, None])


@pytest.mark.parametrize("kv", ["fp16", "fp32"])
# head sizes 64 and 128; 1, 2, 4, 5 query heads per KV head (heads that share a CTA); rows around the 16-row tile; the
# key-split form (few rows) and the shared form (many rows x heads); a context in front of the rows
@pytest.mark.parametrize("heads,kv_heads,D,T,ctx", [(4, 2, 64, 16, 0), (4, 1, 64, 17, 33), (5, 1, 128, 31, 0), (3, 3, 128, 47, 100),
                                                    (4, 1, 128, 129, 7), (16, 4, 64, 640, 0)])
def test_prefill_attention_matches_decode(heads, kv_heads, D, T, ctx, kv):
    """One layer, so that the rows differ only in the attention's summation order: the prefill's last logits and cache
    against a second state fed token by token for the last rows.  A sum that rounds differently may move an int8
    activation by one of 127 steps, about 1e-3 of the logits' spread behind one layer; a wrong key, mask or head is O(1)."""
    cfg = synthetic.toy_config(hidden=heads * D, layers=1, heads=heads, kv_heads=kv_heads, inter=512, vocab=512)
    dm = rt.to_device(synthetic.random_model(cfg, seed=heads * T + D, norm_jitter=0.1))
    toks = [int(t) for t in np.random.default_rng(T).integers(0, cfg.vocab_size, ctx + T)]
    a = rt.init_state(dm, ctx + T, kv_dtype=kv)
    if ctx:
        rt.forward_prefill(dm, a, toks[:ctx])
    got = rt.forward_prefill(dm, a, toks[ctx:])
    b = rt.init_state(dm, ctx + T, kv_dtype=kv)
    for t in toks:
        want = rt.forward_one(dm, b, t)
    assert np.abs(got - want).max() <= 5e-3 * (want.max() - want.min())
    # every other row of the tile through the logits of all rows
    a.pos = ctx
    rows = rt.forward_prefill_all_logits(dm, a, toks[ctx:])
    b.pos = ctx
    for i, t in enumerate(toks[ctx:]):
        want = rt.forward_one(dm, b, t)
        if i % 7 == 0 or i == T - 1:
            assert np.abs(rows[i] - want).max() <= 5e-3 * (want.max() - want.min()), i
    dm.close()


def test_prefill_longer_than_the_row_scratch():
    """More rows than go through the layers at once (2048)."""
    cfg = synthetic.toy_config(hidden=128, layers=1, heads=2, kv_heads=1, inter=256, vocab=256)
    dm = rt.to_device(synthetic.random_model(cfg, seed=5, norm_jitter=0.1))
    toks = [int(t) for t in np.random.default_rng(6).integers(0, cfg.vocab_size, 2100)]
    a, b = rt.init_state(dm, 2110), rt.init_state(dm, 2110)
    got = rt.forward_prefill(dm, a, toks)
    for i in range(0, 2100, 420):
        want = rt.forward_prefill(dm, b, toks[i:i + 420])
    assert a.pos == b.pos == 2100
    assert np.abs(got - want).max() <= 5e-3 * (want.max() - want.min())
    dm.close()
