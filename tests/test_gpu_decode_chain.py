"""The layers of a one-sequence decode step as one kernel against the kernels of a layer, launched one by one (which a forced path of
the products takes): the same arithmetic in the same order, so logits, tokens and cache rows are bit-equal.  Rows whose blocks end
inside a warp's piece, past 256 blocks (a lane's second) and with an odd number of weight chunks; CTAs with none, one and several
row groups; positions around a piece's batches of keys, and the position where a state goes over to launches."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

K = importlib.import_module("litespark_inference_b200.torchless.kernel")
rt = importlib.import_module("litespark_inference_b200.torchless.runtime")
synthetic = importlib.import_module("litespark_inference_b200.torchless.synthetic")

LIMIT = 704        # positions that the one kernel takes
ONE_KERNEL = 4     # embedding, layers, LM head, end of the step


def _both(dm, run):
    """run(state-making function) with the layers as one kernel and as launches."""
    lib, out = K.load_library(), []
    try:
        for path in (0, 1):
            K.check(lib.lspk_linear_force_path(path))
            out.append(run(path == 0))
    finally:
        K.check(lib.lspk_linear_force_path(0))
    return out


def _steps(dm, kv, ctx, n, chained):
    lib = K.load_library()
    path = 0 if chained else 1
    st = rt.init_state(dm, ctx + n, kv_dtype=kv)
    if ctx:
        K.check(lib.lspk_linear_force_path(0))
        rt.prefill_first_token(st, np.random.default_rng(ctx).integers(0, 500, ctx))
        K.check(lib.lspk_linear_force_path(path))
    logits = [rt.forward_one(dm, st, 3 + 7 * i) for i in range(n)]
    assert (st.step_kernel_count == ONE_KERNEL) == (chained and ctx + n <= LIMIT)
    out = logits + list(st.read_kv(dm.config.num_layers - 1, ctx + n))
    st.close()
    return out


@pytest.mark.parametrize("kv", ["fp16", "fp32"])
@pytest.mark.parametrize("family,hidden,heads,kv_heads,inter", [
    ("bitnet", 256, 4, 2, 512), ("falcon", 256, 2, 1, 528), ("bitnet", 1280, 10, 5, 4112), ("falcon", 640, 10, 2, 4672),
    ("bitnet", 2560, 20, 5, 6912), ("bitnet", 2304, 36, 12, 7104)])
def test_steps_equal_those_of_launches(family, hidden, heads, kv_heads, inter, kv):
    make = (synthetic.toy_config, synthetic.random_model) if family == "bitnet" else (synthetic.toy_falcon_config, synthetic.random_falcon_model)
    dm = rt.DeviceModel(make[1](make[0](hidden, 2, heads, kv_heads, inter), seed=5, norm_jitter=0.2))
    for ctx, n in ((0, 3), (30, 4), (253, 5)):
        for a, b in zip(*_both(dm, lambda chained: _steps(dm, kv, ctx, n, chained))):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("kv", ["fp16", "fp32"])
def test_positions_up_to_the_limit_and_past_it(kv):
    dm = rt.DeviceModel(synthetic.random_model(synthetic.toy_config(), seed=6, norm_jitter=0.2))
    for a, b in zip(*_both(dm, lambda chained: _steps(dm, kv, LIMIT - 4, 4, chained))):
        assert np.array_equal(a, b)

    def greedy(chained):
        st = rt.init_state(dm, LIMIT + 40, kv_dtype=kv)
        lib = K.load_library()
        K.check(lib.lspk_linear_force_path(0))
        first = rt.prefill_first_token(st, np.random.default_rng(2).integers(0, 500, LIMIT - 20))
        K.check(lib.lspk_linear_force_path(0 if chained else 1))
        ids = rt.decode_greedy(st, first, 30)                 # over the limit in the middle
        one = [rt.forward_step(st, [ids[-1]])[0]]             # the token id in, the token id out
        st.set_pos(0, LIMIT - 20)                             # and back below it
        again = rt.decode_greedy(st, first, 30)
        st.close()
        assert again == ids
        return ids + [int(one[0])]

    a, b = _both(dm, greedy)
    assert a == b


def test_shapes_that_the_one_kernel_does_not_take():
    """Head dimension 256; more row groups than three per SM; norm weights of 32 bits (none here: bf16 by construction)."""
    sms = K.load_library(True).lspk_sm_count()
    for cfg in (synthetic.toy_config(512, 2, 2, 1, 512), synthetic.toy_config(256, 1, 4, 2, 48 * sms + 64)):
        dm = rt.DeviceModel(synthetic.random_model(cfg, seed=7, fast=True))
        st = rt.init_state(dm, 16)
        assert np.isfinite(rt.forward_one(dm, st, 1)).all() and st.step_kernel_count > ONE_KERNEL
        st.close()
