"""Inference states that are freed and made again, and the LM head's table formats."""
import importlib
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

dev = importlib.import_module("litespark_inference_b200.torchless.device")
K = importlib.import_module("litespark_inference_b200.torchless.kernel")
rt = importlib.import_module("litespark_inference_b200.torchless.runtime")
synthetic = importlib.import_module("litespark_inference_b200.torchless.synthetic")


def test_a_state_made_again_is_a_new_state():
    """A freed state may be handed out again: empty cache, position 0, the same tokens as a fresh one; with another
    shape, after the model's tensors changed, and after the model has gone it is not."""
    cfg = synthetic.toy_config()
    m = synthetic.random_model(cfg, seed=3, norm_jitter=0.1)
    dm = rt.DeviceModel(m)
    prompt = [int(t) for t in np.random.default_rng(1).integers(0, cfg.vocab_size, 20)]
    want = rt.generate(dm, prompt, 10, state=rt.init_state(dm, 64))      # freed here
    for _ in range(3):
        st = rt.init_state(dm, 64)
        assert st.pos == 0
        k, v = st.read_kv(0, 64)
        assert not k.any() and not v.any()
        assert rt.generate(dm, prompt, 10, state=st) == want
        two = rt.init_state(dm, 64)                                      # while the first is in use
        assert rt.generate(dm, prompt, 10, state=two) == want
        st.close()
        two.close()
    other = rt.init_state(dm, 65, kv_dtype="fp32")
    assert rt.generate(dm, prompt, 10, state=other)[0] == want[0]
    other.close()
    # new norm weights: the graph of the parked state must not survive them
    g = np.ascontiguousarray(m.final_norm[::-1])
    K.check(dm.lib.lspk_model_set_norm(dm.handle, -1, 4, g.ctypes.data, 1, g.shape[0]))
    m2 = synthetic.random_model(cfg, seed=3, norm_jitter=0.1)
    m2.final_norm = g
    dm2 = rt.DeviceModel(m2)
    assert rt.generate(dm, prompt, 10, state=rt.init_state(dm, 65, kv_dtype="fp32")) == \
        rt.generate(dm2, prompt, 10, state=rt.init_state(dm2, 65, kv_dtype="fp32"))
    late = rt.init_state(dm2, 64)
    dm2.close()
    late.close()                                                         # its model is gone
    dm.close()


_TRACE_AND_LAUNCH_MODE = """
import ctypes, importlib
import numpy as np
import __graft_entry__ as entry
entry.load_package()
K = importlib.import_module("litespark_inference_b200.torchless.kernel")
rt = importlib.import_module("litespark_inference_b200.torchless.runtime")
synthetic = importlib.import_module("litespark_inference_b200.torchless.synthetic")
dm = rt.DeviceModel(synthetic.random_model(synthetic.toy_config(), seed=3))
lib = dm.lib

def records():
    n, out = ctypes.c_int(), np.zeros((4096, 16), np.uint64)
    K.check(lib.lspk_trace_read(out.ctypes.data, 4096, ctypes.byref(n)))
    return n.value

def free_bytes():
    f = ctypes.c_size_t()
    K.check(lib.lspk_mem_info(ctypes.byref(f), None))
    return f.value

def one_step(st):
    return rt.forward_one(dm, st, 5)

st = rt.init_state(dm, 64)
want = one_step(st)
st.close()                                   # its graph was captured without a trace
K.check(lib.lspk_trace_begin(64))
st = rt.init_state(dm, 64)
assert np.array_equal(one_step(st), want)
per_step = records()
assert per_step > 0
st.close()
K.check(lib.lspk_trace_begin(32))            # fits the buffer: a state made again keeps its graph and records
st = rt.init_state(dm, 64)
assert np.array_equal(one_step(st), want) and records() == per_step
K.check(lib.lspk_trace_begin(2048))          # replaces the buffer under a live state ...
assert rt.forward_one(dm, st, 7).shape == want.shape and records() > 0
st.close()
K.check(lib.lspk_trace_begin(4096))          # ... and under a freed one
st = rt.init_state(dm, 64)
assert np.array_equal(one_step(st), want) and records() > 0
st.close()
st = rt.init_state(dm, 8192, batch=8, kv_dtype="fp32")     # large enough to show in the free memory; parked in its place
held = st.device_bytes
assert held > 50e6
st.close()
before = free_bytes()
K.check(lib.lspk_set_pdl(1))                 # no change: the freed state stays
assert free_bytes() == before
K.check(lib.lspk_set_pdl(0))
assert free_bytes() >= before + held // 2
st = rt.init_state(dm, 8192, batch=8, kv_dtype="fp32")
st.close()
before = free_bytes()
K.check(lib.lspk_linear_force_path(1))       # the kernels of the products are in the graph too
assert free_bytes() >= before + held // 2
K.check(lib.lspk_linear_force_path(0))
st = rt.init_state(dm, 64)
assert np.array_equal(one_step(st), want)
st.close()                                   # a timing harness that turns programmatic launch off while it captures
dev = importlib.import_module("litespark_inference_b200.torchless.device")
w = dev.DeviceWeight(np.full((64, 64), 0x55, np.uint8), 1.0)
x, y, ms = dev.DeviceArray.from_numpy(np.ones(256, np.float32)), dev.DeviceArray((2, 64), np.float32), ctypes.c_float()
K.check(lib.lspk_set_pdl(1))
st = rt.init_state(dm, 64)
one_step(st)
st.close()
K.check(lib.lspk_bench_linear_copies_independent((ctypes.c_void_p * 1)(w.handle), None, 1, x.ptr, y.ptr, 1, 1, 2, 1, ctypes.byref(ms)))
"""


def test_a_state_made_after_a_trace_or_launch_mode_change_uses_it():
    """In a process of its own: the trace buffer stays installed."""
    _in_own_process(_TRACE_AND_LAUNCH_MODE)


_GIVEN_BACK = """
import ctypes, importlib
import numpy as np
import __graft_entry__ as entry
entry.load_package()
name = "litespark_inference_b200.torchless."
K, rt, synthetic = (importlib.import_module(name + n) for n in ("kernel", "runtime", "synthetic"))
dms = [rt.DeviceModel(synthetic.random_model(synthetic.toy_config(), seed=3)) for _ in range(4)]
lib = dms[0].lib

def free_bytes():
    f = ctypes.c_size_t()
    K.check(lib.lspk_mem_info(ctypes.byref(f), None))
    return f.value

big = dict(t_max=8192, batch=24, kv_dtype="fp32")            # 400 MB: two of them are kept, a third takes the first one's place
held = []
for dm in dms:
    st = rt.init_state(dm, **big)
    size = st.device_bytes
    rt.forward_step(st, np.arange(24, dtype=np.int32))
    before = free_bytes()
    st.close()
    held.append(free_bytes() - before < size // 2)
assert 3.9e8 < size < 4.4e8 and held == [True, True, False, False], (size, held)
before = free_bytes()
st = rt.init_state(dms[3], **big)                            # the last one is among those kept
assert free_bytes() == before
st.close()
rt.release_parked_states()
assert free_bytes() - before > 1.9 * size
rt.release_parked_states()                                   # nothing left: no effect
st = rt.init_state(dms[0], **big)
st.close()
K.check(lib.lspk_debug_allocation_limit(1 << 30))            # an allocation of this library that fails takes it back
before = free_bytes()
assert not lib.lspk_malloc(2 << 30)
assert free_bytes() - before > 0.9 * size
"""


def test_memory_of_parked_states_is_bounded_and_given_back():
    _in_own_process(_GIVEN_BACK)


_NO_PINNED = """
import ctypes, importlib
import numpy as np
import __graft_entry__ as entry
entry.load_package()
name = "litespark_inference_b200.torchless."
K, rt, synthetic = (importlib.import_module(name + n) for n in ("kernel", "runtime", "synthetic"))
dm = rt.DeviceModel(synthetic.random_model(synthetic.toy_config(), seed=3))
lib = dm.lib

def free_bytes():
    f = ctypes.c_size_t()
    K.check(lib.lspk_mem_info(ctypes.byref(f), None))
    return f.value

st = rt.init_state(dm, t_max=8192, batch=24, kv_dtype="fp32")
size = st.device_bytes
rt.forward_step(st, np.arange(24, dtype=np.int32))
st.close()                                                   # parked
a, b = np.ones(2560, np.float32), np.full(2560, 2, np.float32)
K.check(lib.lspk_debug_allocation_limit(1000))               # neither a pinned buffer nor device scratch
before = free_bytes()
lib.lspk_clear_error()
lib.add_inplace_fp32_sm100(a, b, a.size)
assert lib.lspk_error_count() >= 1 and (a == 1).all()
assert free_bytes() - before > 0.9 * size                    # parked memory was given back before it failed
K.check(lib.lspk_debug_allocation_limit(0))
lib.lspk_clear_error()
lib.add_inplace_fp32_sm100(a, b, a.size)                     # pinned memory is asked for again: no device scratch was made
before = free_bytes()
K.check(lib.lspk_debug_allocation_limit(1000))
lib.relu2_mul_fp32_batched_sm100(a, b, b, 1, a.size)
assert lib.lspk_error_count() == 0 and (a == 3).all() and (b == 18).all() and free_bytes() == before
"""


def test_small_host_calls_without_pinned_memory():
    _in_own_process(_NO_PINNED)


_SCRATCH_LOST = """
import ctypes, importlib
import numpy as np
import __graft_entry__ as entry
entry.load_package()
name = "litespark_inference_b200.torchless."
K, rt, dev, synthetic, loader = (importlib.import_module(name + n) for n in ("kernel", "runtime", "device", "synthetic", "loader"))
m = synthetic.random_model(synthetic.toy_config(), seed=3)
dm = rt.DeviceModel(m)
lib = dm.lib
toks = np.array([1, 2, 3, 4], np.int32)

def two_steps(t_max=64):
    st = rt.init_state(dm, t_max, batch=4)
    rt.forward_step(st, toks)
    logits = rt.forward_step(st, toks + 9, want_logits=True)[1]
    st.close()
    return logits

want = two_steps()
# a product of many rows that finds no memory: the library's int8 rows are gone, the next step has to make them again
M, Kd = 4096, 1024
w = dev.DeviceWeight(np.full((64, Kd // 4), 0x55, np.uint8), 1.0)
x, y, q = dev.DeviceArray((M, Kd), np.float32), dev.DeviceArray((M, 64), np.float32), dev.DeviceArray((M, Kd), np.int8)
x.fill_bytes(0)
a = K.LinearArgs()
a.w[0], a.out[0], a.n_mats, a.M, a.prologue, a.x_f32, a.xq_out = w.handle, y.ptr, 1, M, K.PRO_QUANT, x.ptr, q.ptr
K.check(lib.lspk_linear_force_path(1))
K.check(lib.lspk_debug_allocation_limit(1 << 20))
assert lib.lspk_linear(ctypes.byref(a)) == 2
K.check(lib.lspk_debug_allocation_limit(0))
K.check(lib.lspk_linear_force_path(0))
assert np.array_equal(two_steps(), want)
# a long cache takes another attention kernel, another table another LM head
assert np.array_equal(two_steps(4000), want)
q8, s8 = loader.quantize_embedding(m.embed_tokens, 127)
K.check(lib.lspk_model_set_lm_head(dm.handle, 1, q8.ctypes.data, s8.ctypes.data))
int8 = two_steps()
assert 0 < np.abs(int8 - want).max() < 0.1 * np.abs(want).max()
"""


_SHORT_OF_MEMORY = """
import importlib
import numpy as np
import __graft_entry__ as entry
entry.load_package()
name = "litespark_inference_b200.torchless."
K, rt, synthetic = (importlib.import_module(name + n) for n in ("kernel", "runtime", "synthetic"))
dm = rt.DeviceModel(synthetic.random_model(synthetic.toy_config(), seed=3, norm_jitter=0.1))
lib = dm.lib
toks = [int(t) for t in np.random.default_rng(1).integers(0, 1024, 1000)]
row = 4 * (3 * 256 + 2 * 128 + 512 + 1)
a, b = rt.init_state(dm, 2048), rt.init_state(dm, 2048)
small = a.device_bytes
want = rt.forward_prefill(dm, a, toks)
assert a.device_bytes == small + (1024 - 128) * row          # as many rows as the prompt, not as the cache could take
K.check(lib.lspk_debug_allocation_limit(1200000))            # the widest buffer finds room for 512 rows
got = rt.forward_prefill(dm, b, toks)
assert b.pos == 1000 and b.device_bytes == small + (512 - 128) * row
# pieces of 512 rows: other attention sums, so as for a prompt given in pieces (test_gpu_prefill_kernels.py)
assert np.abs(got - want).max() <= 5e-3 * (want.max() - want.min())
K.check(lib.lspk_debug_allocation_limit(1000))               # nothing at all: an error, and the state is still good for use
b.pos = 0
try:
    rt.forward_prefill(dm, b, toks)
    raise SystemExit("a prefill without memory went through")
except K.KernelError:
    pass
K.check(lib.lspk_debug_allocation_limit(0))
b.pos = 0
assert np.abs(rt.forward_prefill(dm, b, toks) - want).max() <= 5e-3 * (want.max() - want.min())
assert b.device_bytes == a.device_bytes
"""


def test_a_long_prompt_makes_do_with_less_memory():
    _in_own_process(_SHORT_OF_MEMORY)


def _in_own_process(code):
    r = subprocess.run([sys.executable, "-c", code], cwd=Path(__file__).resolve().parent.parent, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def test_a_step_shape_is_warmed_again_after_scratch_or_tables_changed():
    """In a process of its own, whose scratch no other test has grown."""
    _in_own_process(_SCRATCH_LOST)


@pytest.mark.parametrize("kind", [0, 1, 2])
# one row (pairs of table rows per warp), the tensor-core tiles at 2, 8, 9, 17 rows; hidden sizes on and off its K step;
# an odd vocabulary
@pytest.mark.parametrize("T,H", [(1, 2560), (1, 96), (2, 128), (8, 2560), (9, 256), (17, 640), (3, 96)])
def test_lm_head_formats(kind, T, H):
    rng = np.random.default_rng(kind * 100 + T)
    V = 1037
    x = (rng.standard_normal((T, H)) * np.exp(rng.uniform(-3, 3, (T, 1)))).astype(np.float32)
    sc = rng.uniform(0.5, 1.5, V).astype(np.float32)
    if kind == 0:
        table = (rng.standard_normal((V, H)).astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
        vals = (table.astype(np.uint32) << 16).view(np.float32).astype(np.float64)
    elif kind == 1:
        table = rng.integers(-128, 128, (V, H)).astype(np.int8)
        vals = table.astype(np.float64) * sc[:, None]
    else:
        table = rng.integers(0, 256, (V, H // 2)).astype(np.uint8)
        n = np.stack([table & 15, table >> 4], axis=-1).reshape(V, H).astype(np.int64)
        vals = (n - 16 * (n > 7)).astype(np.float64) * sc[:, None]
    de, ds, dx = dev.DeviceArray.from_numpy(table), dev.DeviceArray.from_numpy(sc), dev.DeviceArray.from_numpy(x)
    dl = dev.DeviceArray((T, V), np.float32)
    K.check(K.load_library().lspk_lm_head(kind, de.ptr, ds.ptr if kind else None, dx.ptr, dl.ptr, T, V, H))
    want = x.astype(np.float64) @ vals.T
    # fp32 sums of H products in any order: H * 2^-24 of the sum of their magnitudes at the very most
    bound = H * 2.0**-24 * (np.abs(x).astype(np.float64) @ np.abs(vals).T) + 1e-30
    assert (np.abs(dl.numpy() - want) <= bound).all()


@pytest.mark.parametrize("kind", [0, 1, 2])
# rows whose three 16-bit terms are the longest that fit the tensor-core kernel and the next longer, a wide model's hidden
# size, the widest that the eight rows of the other kernel fit; more rows than its CTAs take
@pytest.mark.parametrize("T,H", [(8, 4224), (2, 4352), (2, 5120), (8, 5120), (9, 5120), (2, 25600), (8, 6400), (1190, 128)])
def test_lm_head_rows_of_any_width(kind, T, H):
    rng = np.random.default_rng(H + T)
    V = 67
    x = rng.standard_normal((T, H)).astype(np.float32)
    sc = rng.uniform(0.5, 1.5, V).astype(np.float32)
    if kind == 0:
        table = (rng.standard_normal((V, H)).astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
        vals = (table.astype(np.uint32) << 16).view(np.float32).astype(np.float64)
    elif kind == 1:
        table = rng.integers(-128, 128, (V, H)).astype(np.int8)
        vals = table * sc.astype(np.float64)[:, None]
    else:
        table = rng.integers(0, 256, (V, H // 2)).astype(np.uint8)
        n = np.stack([table & 15, table >> 4], axis=-1).reshape(V, H).astype(np.int64)
        vals = (n - 16 * (n > 7)) * sc.astype(np.float64)[:, None]
    de, ds, dx = dev.DeviceArray.from_numpy(table), dev.DeviceArray.from_numpy(sc), dev.DeviceArray.from_numpy(x)
    dl = dev.DeviceArray((T, V), np.float32)
    K.check(K.load_library().lspk_lm_head(kind, de.ptr, ds.ptr if kind else None, dx.ptr, dl.ptr, T, V, H))
    # as in test_lm_head_formats
    bound = H * 2.0**-24 * (np.abs(x).astype(np.float64) @ np.abs(vals).T)
    assert (np.abs(dl.numpy() - x.astype(np.float64) @ vals.T) <= bound).all()


@pytest.mark.parametrize("table", ["bf16", "int8", "int4"])
def test_batched_decode_of_a_wide_model(table):
    """A hidden size beyond the tensor-core LM head: the greedy choice of several sequences comes from a row argmax."""
    cfg = synthetic.toy_config(hidden=5120, layers=1, heads=40, kv_heads=8, inter=256, vocab=256)
    m = synthetic.random_model(cfg, seed=2, norm_jitter=0.1)
    loader = importlib.import_module("litespark_inference_b200.torchless.loader")
    if table != "bf16":
        q, m.embed_scale = loader.quantize_embedding(m.embed_tokens, 127 if table == "int8" else 7)
        setattr(m, "embed_" + table, q)
        m.embed_tokens = None
    dm = rt.DeviceModel(m)
    st = rt.init_state(dm, 32, batch=2)
    toks = np.array([3, 77], np.int32)
    for _ in range(4):
        nxt, logits = rt.forward_step(st, toks, want_logits=True)
        assert list(nxt) == [int(np.argmax(r)) for r in logits]
        toks = nxt
    ids = np.empty((3, 2), np.int32)
    K.check(dm.lib.lspk_decode_greedy(st.handle, toks.ctypes.data, 3, ids.ctypes.data))
    st.close()
    rows = rt.forward_prefill_all_logits(dm, rt.init_state(dm, 32), [1, 2, 3, 4, 5])
    assert np.isfinite(rows).all()
    dm.close()


@pytest.mark.parametrize("kind", [1, 2])
@pytest.mark.parametrize("T,H", [(2, 256), (8, 2560), (9, 640), (16, 2560), (2, 4096)])
def test_lm_head_rows_as_accurate_as_one_row(kind, T, H):
    """The tensor-core form for several rows against the one-row kernel (fp32 multiply-adds): as close to float64."""
    rng = np.random.default_rng(kind * 10 + H)
    V = 2003
    x = rng.standard_normal((T, H)).astype(np.float32)
    if kind == 1:
        table = rng.integers(-128, 128, (V, H)).astype(np.int8)
        vals = table.astype(np.float64)
    else:
        table = rng.integers(0, 256, (V, H // 2)).astype(np.uint8)
        n = np.stack([table & 15, table >> 4], axis=-1).reshape(V, H).astype(np.int64)
        vals = (n - 16 * (n > 7)).astype(np.float64)
    de, ds = dev.DeviceArray.from_numpy(table), dev.DeviceArray.from_numpy(np.ones(V, np.float32))

    def logits(rows):
        dx, dl = dev.DeviceArray.from_numpy(rows), dev.DeviceArray((rows.shape[0], V), np.float32)
        K.check(K.load_library().lspk_lm_head(kind, de.ptr, ds.ptr, dx.ptr, dl.ptr, rows.shape[0], V, H))
        return dl.numpy()

    want = x.astype(np.float64) @ vals.T
    norm = np.sqrt(x.astype(np.float64) ** 2 @ (vals ** 2).T)
    err = [np.sqrt(np.mean(((got - want) / norm) ** 2)) for got in (logits(x), np.concatenate([logits(r[None]) for r in x]))]
    # the one-row sums round H / 32 times per lane and five times across lanes; tensor-core sums of 48 products truncate
    # once each, and some dozens of them are added: no more, up to the scatter of two rounding patterns
    assert err[0] <= 1.15 * err[1], err
    # an fp32 sum of products of these magnitudes, within a few units in the last place of its norm
    assert err[0] <= 4 * 2.0**-24
