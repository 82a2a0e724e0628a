"""Decode attention of several sequences (cache rows fetched once for the query heads of a KV head) against the
one-sequence kernel: the same sums in the same order, so the K and V rows that later layers write are the same to the
bit.  Context lengths around the ends of key batches (8 ranks x key groups x 8 keys), several group sizes, both head sizes."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

rt = importlib.import_module("litespark_inference_b200.torchless.runtime")
synthetic = importlib.import_module("litespark_inference_b200.torchless.synthetic")


@pytest.mark.parametrize("heads,kv_heads,head_dim,lens,t_max,kv", [
    (8, 2, 128, (511, 1100), 1120, "fp32"),          # around one batch (512 keys), into a third
    (8, 2, 128, (1, 1021, 1030), 2100, "fp16"),      # a sequence with a key in one rank only; around one batch (1024 keys)
    (4, 2, 64, (5, 1025, 257, 64), 1100, "fp32"),    # head size 64, two heads per KV head
    (8, 1, 64, (33, 2050), 2100, "fp16"),            # eight heads per KV head: four CTAs of two
    (6, 3, 128, (300, 31, 2), 600, "fp32"),          # barely long enough
    (3, 1, 128, (300, 31), 600, "fp32"),             # an odd group: one head per CTA
])
def test_grouped_heads_equal_single_sequence(heads, kv_heads, head_dim, lens, t_max, kv):
    cfg = synthetic.toy_config(hidden=heads * head_dim, layers=3, heads=heads, kv_heads=kv_heads)
    m = synthetic.random_model(cfg, seed=5, norm_jitter=0.1)
    dm = rt.to_device(m)
    rng = np.random.default_rng(heads)
    steps = 4
    prompts = [np.ascontiguousarray(rng.integers(0, cfg.vocab_size, n), dtype=np.int32) for n in lens]
    forced = rng.integers(0, cfg.vocab_size, (steps, len(lens))).astype(np.int32)
    st = rt.init_state(dm, t_max, batch=len(lens), kv_dtype=kv)
    for b, p in enumerate(prompts):
        assert st.lib.lspk_forward_prefill(st.handle, b, p.ctypes.data, int(p.size), None, None, None) == 0
    for i in range(steps):
        rt.forward_step(st, forced[i], want_logits=True)
    together = [[st.read_kv(li, lens[b] + steps, seq=b) for li in range(cfg.num_layers)] for b in range(len(lens))]
    st.close()
    for b, p in enumerate(prompts):
        s1 = rt.init_state(dm, t_max, kv_dtype=kv)
        rt.forward_prefill(dm, s1, [int(t) for t in p])
        for i in range(steps):
            rt.forward_one(dm, s1, int(forced[i, b]))
        for li in range(cfg.num_layers):
            k1, v1 = s1.read_kv(li, lens[b] + steps)
            assert np.array_equal(k1, together[b][li][0]) and np.array_equal(v1, together[b][li][1]), (b, li)
        s1.close()
    dm.close()


@pytest.mark.parametrize("kv,lens,t_max", [
    ("fp32", (295, 293, 296, 291), 2048),            # in the middle of the steps below the two forms change
    ("fp16", (760, 754, 757, 762, 745), 1000),
    ("fp32", (20, 20, 20, 20, 20, 20, 20, 818), 900),   # one long among short
    ("fp32", (100, 294), 500),                       # two sequences, uneven
    ("fp16", (1994, 40), 2100),
    ("fp16", (5, 9), 4000),                          # a long cache with short sequences
])
def test_steps_across_the_change_of_form(kv, lens, t_max):
    """The form follows the positions, step by step: host-driven steps, a greedy loop over the change, and each sequence
    alone give the same cache rows to the bit (the first two the same tokens)."""
    cfg = synthetic.toy_config(hidden=8 * 128, layers=2, heads=8, kv_heads=2)
    dm = rt.to_device(synthetic.random_model(cfg, seed=6, norm_jitter=0.1))
    rng = np.random.default_rng(len(lens))
    steps, B = 14, len(lens)
    prompts = [np.ascontiguousarray(rng.integers(0, cfg.vocab_size, n), dtype=np.int32) for n in lens]
    first = rng.integers(0, cfg.vocab_size, B).astype(np.int32)

    def state():
        st = rt.init_state(dm, t_max, batch=B, kv_dtype=kv)
        for b, p in enumerate(prompts):
            assert st.lib.lspk_forward_prefill(st.handle, b, p.ctypes.data, int(p.size), None, None, None) == 0
        return st

    one, two = state(), state()
    toks, fed = first, []
    for _ in range(steps):
        fed.append(toks)
        toks = rt.forward_step(one, toks)
    ids = np.empty((steps, B), np.int32)
    assert two.lib.lspk_decode_greedy(two.handle, first.ctypes.data, steps, ids.ctypes.data) == 0
    assert np.array_equal(ids[:-1], np.array(fed[1:])) and np.array_equal(ids[-1], toks)
    for b, p in enumerate(prompts):
        alone = rt.init_state(dm, t_max, kv_dtype=kv)
        rt.forward_prefill(dm, alone, [int(t) for t in p])
        for i in range(steps):
            rt.forward_one(dm, alone, int(fed[i][b]))
        for li in range(cfg.num_layers):
            want = alone.read_kv(li, lens[b] + steps)
            for st in (one, two):
                got = st.read_kv(li, lens[b] + steps, seq=b)
                assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), (b, li)
        alone.close()
    # going back to short positions goes back to the other form
    for b in range(B):
        two.set_pos(b, 3)
        one.set_pos(b, 3)
    assert np.array_equal(rt.forward_step(one, first), rt.forward_step(two, first))
    one.close()
    two.close()
    dm.close()
