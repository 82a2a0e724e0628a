"""The prefill attention by itself, on its own rotated queries and cached rows: against float64, and its error against that
of the kernel which takes fewer than sixteen rows (fp32 multiply-adds, probabilities normalised in front of the values)."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

dev = importlib.import_module("litespark_inference_b200.torchless.device")
K = importlib.import_module("litespark_inference_b200.torchless.kernel")
abi = importlib.import_module("litespark_inference_b200.torchless._runtime_abi")
ops = importlib.import_module("litespark_inference_b200.torchless.ops")


class Attention:
    """Device arrays of one layer: ``ctx`` cached positions and T rows behind them."""

    def __init__(self, Q, KV, D, T, ctx, kv, spread=4.0, seed=0):
        lib = K.load_library()
        fn = lib.lspk_debug_prefill_attention
        fn.argtypes, fn.restype = abi.SIGNATURES["lspk_debug_prefill_attention"]
        self.fn, self.Q, self.KV, self.D, self.T, self.ctx, self.fp16 = fn, Q, KV, D, T, ctx, int(kv == "fp16")
        rng = np.random.default_rng(seed + T + D)
        dt = np.float16 if kv == "fp16" else np.float32
        self.q = (spread * rng.standard_normal((T, Q, D))).astype(np.float32)
        self.k, self.v = (rng.standard_normal((T, KV, D)).astype(np.float32) for _ in range(2))
        self.ck, self.cv = (np.concatenate([rng.standard_normal((ctx, KV, D)), np.full((T, KV, D), 77.0)]).astype(dt) for _ in range(2))
        self.rope = [dev.DeviceArray.from_numpy(a) for a in ops.rope_tables(D, ctx + T, 500000.0)]

    def run(self, block):
        """The rows in calls of ``block``: (output, rotated queries, cached keys, cached values)."""
        put = dev.DeviceArray.from_numpy
        q, k, v, ck, cv, out = put(self.q), put(self.k), put(self.v), put(self.ck), put(self.cv), put(np.zeros_like(self.q))
        pos = dev.DeviceArray.from_numpy(np.arange(self.ctx, self.ctx + self.T, dtype=np.int32))
        for t in range(0, self.T, block):
            n = min(block, self.T - t)
            qo, ko = 4 * t * self.Q * self.D, 4 * t * self.KV * self.D
            K.check(self.fn(q.ptr + qo, k.ptr + ko, v.ptr + ko, ck.ptr, cv.ptr, self.rope[0].ptr, self.rope[1].ptr,
                            pos.ptr + 4 * t, out.ptr + qo, n, self.Q, self.KV, self.D, self.ctx + self.T, self.fp16))
        return out.numpy(), q.numpy(), ck.numpy(), cv.numpy()

    def exact(self, q, ck, cv):
        want = np.empty(q.shape)
        hidden = np.arange(self.ctx + self.T)[None, :] > (self.ctx + np.arange(self.T))[:, None]
        for h in range(self.Q):
            s = q[:, h].astype(np.float64) @ ck[:, h // (self.Q // self.KV)].astype(np.float64).T / np.sqrt(self.D)
            s[hidden] = -np.inf
            p = np.exp(s - s.max(axis=1, keepdims=True))
            want[:, h] = (p / p.sum(axis=1, keepdims=True)) @ cv[:, h // (self.Q // self.KV)].astype(np.float64)
        return want


@pytest.mark.parametrize("kv", ["fp16", "fp32"])
# one row tile and its edges, the key-split form, the shared form (long prompts over many heads) with and without a context
@pytest.mark.parametrize("Q,KV,D,T,ctx", [(4, 1, 128, 16, 0), (5, 5, 64, 33, 200), (20, 5, 128, 128, 0), (20, 5, 128, 700, 77),
                                          (20, 5, 128, 1531, 0), (12, 6, 64, 900, 0)])
@pytest.mark.parametrize("spread", [1.0, 4.0])
def test_no_less_accurate_than_fp32_multiply_adds(Q, KV, D, T, ctx, kv, spread):
    a = Attention(Q, KV, D, T, ctx, kv, spread)
    got, q, ck, cv = a.run(T)
    plain, q2, ck2, cv2 = a.run(8)
    assert np.array_equal(q, q2) and np.array_equal(ck, ck2) and np.array_equal(cv, cv2)
    want = a.exact(q, ck, cv)
    err, ref = (np.linalg.norm(x - want) / np.linalg.norm(want) for x in (got, plain))
    print(f"{Q}/{KV}x{D} T {T} ctx {ctx} {kv} spread {spread}: {err:.3e}, fp32 multiply-adds {ref:.3e}")
    # a score is a sum of D products below |q| |k| of about 4 D at the larger spread, an error of a few 2^-24 of it in the
    # exponent: below 2^-20 of the result, which a lost term of a 16-bit split (2^-12 and more of a product) is not
    assert err <= 2.0**-20
    # two roundings of the same sums: equal up to their scatter
    assert err <= 1.1 * ref + 2e-8


@pytest.mark.parametrize("kv", ["fp16", "fp32"])
# the key-split form and the shared form; 40 rows: a last tile that is not full
@pytest.mark.parametrize("Q,KV,D,T,ctx", [(4, 2, 128, 40, 9), (5, 1, 64, 33, 0), (20, 5, 128, 520, 0), (12, 6, 64, 640, 20)])
@pytest.mark.parametrize("what", ["value", "nan value", "key", "query", "context value", "huge values"])
def test_values_that_are_not_finite_stay_where_they_belong(Q, KV, D, T, ctx, kv, what):
    """An infinite or missing value, key or query element reaches the rows that attend to it and no other, as in the kernel
    for fewer rows, which never touches a masked key."""
    a = Attention(Q, KV, D, T, ctx, kv, spread=1.0)
    at = T - 7                                     # a row of the last tiles: masked for the rows in front of it
    if what == "value":
        a.v[at, 0, 3] = 1e6 if kv == "fp16" else np.inf            # an fp16 cache overflows at 65504
    elif what == "nan value":
        a.v[at, KV - 1, D - 1] = np.nan
    elif what == "key":                            # scores of -inf switch the key off, of +inf and NaN spoil the row
        a.k[at, 0, 5] = np.inf
    elif what == "query":
        a.q[at, Q - 1, 0] = -np.inf
    elif what == "context value":
        if not ctx:
            pytest.skip("no context")
        a.cv[2, 0, 1] = np.inf                     # for every row
    else:
        if kv == "fp16":
            pytest.skip("fp16 values do not reach the end of fp32")
        a.v[:, 0, 0] = 2e38                        # sums of unnormalised probabilities would leave fp32
        a.cv[:, 0, 0] = 2e38
    got, _, ck, cv = a.run(T)
    want, _, ck2, cv2 = a.run(8)
    assert np.array_equal(ck, ck2, equal_nan=True) and np.array_equal(cv, cv2, equal_nan=True)
    if what != "huge values":
        assert not np.isfinite(want).all()
    assert np.isfinite(want[:at]).all() or what == "context value"
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))
    ok = np.isfinite(want)
    assert np.array_equal(np.sign(got[np.isinf(got)]), np.sign(want[np.isinf(want)]))
    scale = np.abs(want[ok]).max() if what == "huge values" else 1.0
    # two roundings of the same sums of values of order 1 (of the largest)
    assert np.abs(got[ok] / scale - want[ok] / scale).max() <= 2.0**-18


@pytest.mark.parametrize("kv", ["fp16", "fp32"])
# four, two and one warps per row tile by the CTAs they make (20 heads x 128 rows: two), and heads that share no key rows in pairs
@pytest.mark.parametrize("Q,KV,D,T,ctx", [(20, 5, 128, 112, 3), (20, 5, 128, 129, 0), (20, 5, 128, 177, 0), (3, 1, 64, 1025, 40),
                                          (25, 5, 128, 513, 0), (40, 5, 128, 900, 0), (7, 7, 64, 1040, 0)])
def test_every_split_of_the_rows_and_keys(Q, KV, D, T, ctx, kv):
    a = Attention(Q, KV, D, T, ctx, kv, 6.0)
    got, q, ck, cv = a.run(T)
    plain, _, _, _ = a.run(8)
    want = a.exact(q, ck, cv)
    err, ref = (np.linalg.norm(x - want) / np.linalg.norm(want) for x in (got, plain))
    assert err <= 1.1 * ref + 2e-8                 # as above: two roundings of the same sums
