"""The workloads whose speed is tracked, at the BitNet-2B and hybrid shapes of ``torchless/synthetic.py`` and
``torchless/hybrid.py``, each through the entry points a program of this package calls:

  linear      ``device.linear`` on device-resident rows: the q/k/v products or an MLP block (gate + up, down)
  gemv_batch  ``lspk_linear_batch``: many independent one-row products in one launch
  host_mlp    an MLP block through the host-array wrappers of ``kernel.py`` (the drop-in boundary), weights registered
  decode      decode steps of 1..8 sequences behind a context (on-device greedy loop, or logits to the host each step)
  prefill     a prompt through ``forward_prefill`` / ``forward_prefill_all_logits``
  generate    one request through the ``BitNet`` facade (state creation, prefill, decode)
  hybrid      a request on a kept hybrid (Mamba-2 + MoE) state: reset, prompt, greedy steps

Weights are seeded and made once per process, as a serving program has them; a case's seed makes its inputs (prompts,
rows).  Ternary weights are uniform over {-1, 0, +1}; per-tensor scales are U(0.5, 1.5) over the gain of such a
matrix, the two projections that write the residual stream another 1 / sqrt(2 * layers) and a quarter below that, so
that attention scores and the residual stream have the spread of a trained network and not that of a saturated one.
The LM head holds the embedding rows in another order, which gives the peaked next-token distribution of a trained
model: a greedy sequence then walks a permutation of the vocabulary instead of deciding ties of noise.
"""
import ctypes
import math

import numpy as np
import torch

import __graft_entry__ as _entry

_entry.load_package()
from litespark_inference_b200.torchless import api, device, hybrid, kernel, model, runtime, tokenizer  # noqa: E402
from litespark_inference_b200.torchless.synthetic import BITNET_2B, BITNET_2B_SHAPES  # noqa: E402

H, I, V = BITNET_2B["hidden_size"], BITNET_2B["intermediate_size"], BITNET_2B["vocab_size"]
LAYERS, HEADS, KV_HEADS = BITNET_2B["num_layers"], BITNET_2B["num_heads"], BITNET_2B["num_kv_heads"]
D = H // HEADS
KV = KV_HEADS * D
EPS = BITNET_2B["rms_norm_eps"]
LAYER_WEIGHTS = sum(n * k for n, k in BITNET_2B_SHAPES.values())
TABLE_BYTES = {"bf16": 2.0, "int8": 1.0, "int4": 0.5}

HYBRID = hybrid.HybridConfig()


# ---- the cases ----------------------------------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: one token's q/k/v products with norm and quantiser fused, as a host-driven layer loop makes it
        {"name": "linear qkv 1 row", "kind": "linear", "block": "qkv", "rows": 1},
        # the largest row count of the layer-shape sweep: an MLP block of a 512-token prompt
        {"name": "linear mlp 512 rows", "kind": "linear", "block": "mlp", "rows": 512},
        # the GEMV bandwidth figure: the gate matrices of a whole model, independent of one another
        {"name": "gemv batch 30 gate", "kind": "gemv_batch", "shape": "gate", "count": 30},
        # a host runtime that keeps its arrays in numpy and calls the kernels one by one, as the reference's does
        {"name": "host mlp 1 row", "kind": "host_mlp", "rows": 1},
        # the headline: one sequence decoding behind a 128-token prompt, fp16 cache, bf16 table
        {"name": "decode 1 ctx 128", "kind": "decode", "family": "bitnet", "table": "bf16", "kv": "fp16", "batch": 1,
         "ctx": 128, "steps": 32, "logits": False},
        # serving: eight sequences of unequal lengths in lock step
        {"name": "decode 8 ctx 128-205", "kind": "decode", "family": "bitnet", "table": "bf16", "kv": "fp16", "batch": 8,
         "ctx": 128, "steps": 16, "logits": False},
        # two long chats whose sampler wants the logits of every step, fp32 cache (the reference's), int8 table
        {"name": "decode 2 ctx 1989 logits", "kind": "decode", "family": "bitnet", "table": "int8", "kv": "fp32", "batch": 2,
         "ctx": 1989, "steps": 8, "logits": True},
        # the headline's prompt
        {"name": "prefill 128", "kind": "prefill", "family": "bitnet", "table": "bf16", "kv": "fp16", "tokens": 128,
         "ctx": 0, "all": False},
        # a long document, of no round length
        {"name": "prefill 1531", "kind": "prefill", "family": "bitnet", "table": "bf16", "kv": "fp16", "tokens": 1531,
         "ctx": 0, "all": False},
        # a short question to the facade with its default int4 table: the whole request, its state included
        {"name": "generate 29 + 24 int4", "kind": "generate", "table": "int4", "prompt": 29, "new": 24, "speculative": False},
        # the hybrid decoder, one request and a batch of sixteen
        {"name": "hybrid 1", "kind": "hybrid", "batch": 1, "prompt": 8, "steps": 23},
        {"name": "hybrid 16", "kind": "hybrid", "batch": 16, "prompt": 8, "steps": 15},
    ]


def _log_int(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi], odd and even alike."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "gemv_batch", "host_mlp", "decode", "decode", "prefill", "prefill", "generate", "hybrid"])
    if kind == "linear":
        return {"kind": kind, "block": rng.choice(["qkv", "mlp"]), "rows": _log_int(rng, 1, 512)}
    if kind == "gemv_batch":
        return {"kind": kind, "shape": rng.choice(["q", "k", "gate", "down"]), "count": rng.randint(2, 30)}
    if kind == "host_mlp":
        return {"kind": kind, "rows": _log_int(rng, 1, 64)}
    family = rng.choice(["bitnet", "bitnet", "falcon"])
    table = "bf16" if family == "falcon" else rng.choice(["bf16", "int8", "int4"])
    kv = rng.choice(["fp16", "fp16", "fp32"])
    if kind == "decode":
        batch = rng.randint(1, 8)
        return {"kind": kind, "family": family, "table": table, "kv": kv, "batch": batch,
                "ctx": _log_int(rng, 16, 4000 // batch), "steps": rng.randint(4, 16), "logits": rng.random() < 0.4}
    if kind == "prefill":
        if rng.random() < 0.3:      # the candidates of a speculative step, checked behind a context
            return {"kind": kind, "family": family, "table": table, "kv": kv, "tokens": rng.randint(2, 8),
                    "ctx": _log_int(rng, 16, 1024), "all": True}
        return {"kind": kind, "family": family, "table": table, "kv": kv, "tokens": _log_int(rng, 9, 1531), "ctx": 0,
                "all": False}
    if kind == "generate":
        return {"kind": kind, "table": rng.choice(["bf16", "int4"]), "prompt": _log_int(rng, 6, 400), "new": rng.randint(4, 32),
                "speculative": rng.random() < 0.4}
    return {"kind": kind, "batch": rng.randint(1, 16), "prompt": rng.randint(2, 8), "steps": rng.randint(4, 15)}


# ---- weights, made once per process -------------------------------------------------------------------------------
_TRITS = np.array([a | (b << 2) | (c << 4) | (d << 6) for d in range(3) for c in range(3) for b in range(3)
                   for a in range(3)], dtype=np.uint8)
_kept = {}


def _keep(key, make):
    if key not in _kept:
        _kept[key] = make()
    return _kept[key]


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _packed(g, n, k, copies=None):
    """Packed bytes [n, k/4] (or [copies, n * k/4]) of uniform ternary weights; 81 byte values hold four trits each."""
    shape = (n, k // 4) if copies is None else (copies, n * (k // 4))
    at = torch.randint(0, 81, shape, generator=g, device="cuda", dtype=torch.uint8)
    return torch.from_numpy(_TRITS).cuda()[at.int()].cpu().numpy()


def _scale(g, k, branch_layers=0):
    s = (0.5 + torch.rand((), generator=g, device="cuda").item()) * math.sqrt(1.5 / k)
    return float(np.float32(s * (0.25 / math.sqrt(2 * branch_layers)) if branch_layers else s))


def _projection(g, n, k, branch_layers=0):
    return model.PackedProjection(w_packed=_packed(g, n, k), w_sum=None, scale=_scale(g, k, branch_layers), in_features=k,
                                  out_features=n)


def _bf16_bits(t):
    return t.to(torch.bfloat16).view(torch.int16).cpu().numpy().view(np.uint16)


def _gamma(g, *shape):
    return _bf16_bits(1.0 + 0.1 * (2.0 * torch.rand(shape, generator=g, device="cuda") - 1.0))


def _table(g, kind, v, h):
    """(table, permuted table) as device tensors plus their row scales: the embedding and the LM head."""
    if kind == "bf16":
        t, s = torch.randn((v, h), generator=g, device="cuda").to(torch.bfloat16).view(torch.int16), None
    elif kind == "int8":
        t = (torch.randn((v, h), generator=g, device="cuda") * 32.0).round_().clamp_(-127, 127).to(torch.int8)
        s = (0.9 + 0.2 * torch.rand(v, generator=g, device="cuda")) / 32.0
    else:
        t = torch.randint(0, 256, (v, h // 2), generator=g, device="cuda", dtype=torch.uint8)
        s = (0.9 + 0.2 * torch.rand(v, generator=g, device="cuda")) / 4.6
    order = torch.randperm(v, generator=g, device="cuda")
    host = lambda x: None if x is None else (x.cpu().numpy().view(np.uint16) if x.dtype == torch.int16 else x.cpu().numpy())  # noqa: E731
    return (host(t), host(s)), (host(t[order]), host(None if s is None else s[order])), order.cpu().numpy()


def _build_model(family, table):
    g = _generator(20 + 3 * (family == "falcon") + ["bf16", "int8", "int4"].index(table))
    (emb, emb_s), (head, head_s), order = _table(g, table, V, H)
    layers = []
    for _ in range(LAYERS):
        p = dict(q_proj=_projection(g, H, H), k_proj=_projection(g, KV, H), v_proj=_projection(g, KV, H),
                 o_proj=_projection(g, H, H, LAYERS), gate_proj=_projection(g, I, H), up_proj=_projection(g, I, H),
                 down_proj=_projection(g, H, I, LAYERS), input_norm=_gamma(g, H), post_attn_norm=_gamma(g, H))
        if family == "bitnet":
            layers.append(model.PackedLayer(**p, attn_sub_norm=_gamma(g, H), ffn_sub_norm=_gamma(g, I)))
        else:
            layers.append(model.PackedFalconLayer(**p))
    if family == "bitnet":
        m = model.PackedBitNetModel(config=model.BitNetConfig(**BITNET_2B), embed_tokens=None, final_norm=_gamma(g, H), layers=layers)
    else:
        m = model.PackedFalconModel(config=model.FalconTernaryConfig(**BITNET_2B), embed_tokens=None, final_norm=_gamma(g, H),
                                    layers=layers)
    field = {"bf16": "tokens", "int8": "int8", "int4": "int4"}[table]
    setattr(m, "embed_" + field, emb)
    m.embed_scale = emb_s
    for f in ("tokens", "int8", "int4"):
        setattr(m, "lm_head_" + f, head if f == field else None)
    m.lm_head_scale = head_s
    follows = np.empty(V, np.int64)      # the token whose head row is a token's embedding row
    follows[order] = np.arange(V)
    torch.cuda.empty_cache()
    return runtime.DeviceModel(m), follows


def _device_model(family, table):
    return _keep(("model", family, table), lambda: _build_model(family, table))


def _build_hybrid():
    c, g = HYBRID, _generator(40)
    di, conv = c.nheads * c.headdim, c.nheads * c.headdim + 2 * c.d_state
    u = lambda lo, hi, *shape: (lo + (hi - lo) * torch.rand(shape, generator=g, device="cuda")).cpu().numpy()  # noqa: E731
    layers = []
    for li in range(c.num_layers):
        if li % 2 == 0:
            layers.append(hybrid.MambaLayer(
                kind="mamba", norm=_gamma(g, H), in_proj=_projection(g, 2 * di + 2 * c.d_state + c.nheads, H),
                out_proj=_projection(g, H, di, c.num_layers), conv_w=u(-0.5, 0.5, conv, c.conv_width), conv_b=u(-0.1, 0.1, conv),
                A=-np.exp(u(-4.0, 0.0, c.nheads)), dt_bias=u(-4.0, -2.0, c.nheads), D=np.ones(c.nheads, np.float32),
                gated_norm=_gamma(g, di), nheads=c.nheads, headdim=c.headdim, d_state=c.d_state))
        else:
            e = c.num_experts
            scales = [[_scale(g, H), _scale(g, H), _scale(g, I, c.num_layers)] for _ in range(e)]
            layers.append(hybrid.MoELayer(
                kind="moe", norm=_gamma(g, H), router=(0.02 * torch.randn((e, H), generator=g, device="cuda")).cpu().numpy(),
                experts_packed=_packed(g, I, H, 3 * e).reshape(e, 3, -1), scales=np.array(scales, np.float32),
                sub_norm=_gamma(g, e, I), hidden_size=H, intermediate_size=I))
    emb = _bf16_bits(torch.randn((V, H), generator=g, device="cuda"))
    torch.cuda.empty_cache()
    return hybrid.DeviceHybrid(hybrid.HybridModel(config=c, embed_tokens=emb, final_norm=_gamma(g, H), layers=layers))


def _device_weight(shape, copy):
    def make():
        n, k = BITNET_2B_SHAPES[shape]
        g = _generator(1000 + 100 * list(BITNET_2B_SHAPES).index(shape) + copy)
        return device.DeviceWeight(_packed(g, n, k), _scale(g, k))
    return _keep(("weight", shape, copy), make)


def _host_weight(shape):
    def make():
        n, k = BITNET_2B_SHAPES[shape]
        g = _generator(2000 + list(BITNET_2B_SHAPES).index(shape))
        w = _packed(g, n, k)
        kernel.register_packed(w)
        return w, _scale(g, k)
    return _keep(("host weight", shape), make)


# ---- inputs ---------------------------------------------------------------------------------------------------------
class _View:
    """A DeviceArray as torch sees it."""

    def __init__(self, a):
        self.a = a
        self.__cuda_array_interface__ = {"shape": a.shape, "typestr": a.dtype.str, "data": (a.ptr, False), "version": 3}


def _tensor(a):
    return torch.as_tensor(_View(a), device="cuda")


def _normal(g, *shape):
    return torch.randn(shape, generator=g, device="cuda").cpu().numpy()


class _HybridState(hybrid.HybridState):
    def __del__(self):
        self.close()


def prepare(case, seed):
    g = _generator(seed)
    rng = np.random.default_rng(seed)
    s = dict(case)
    kind = case["kind"]
    if kind == "linear":
        m = case["rows"]
        s["x"] = device.DeviceArray.from_numpy(_normal(g, m, H))
        s["gamma"] = device.DeviceArray.from_numpy(_gamma(g, H))
        names = ("q", "k", "v") if case["block"] == "qkv" else ("gate", "up")
        s["w"] = [_device_weight(n, 0) for n in names]
        s["out"] = [device.DeviceArray((m, w.N), np.float32) for w in s["w"]]
        if case["block"] == "mlp":
            s["gamma2"] = device.DeviceArray.from_numpy(_gamma(g, I))
            s["down"] = _device_weight("down", 0)
            s["out"] = [s["out"][0], None]
            s["y"] = device.DeviceArray((m, H), np.float32)
        s["views"] = [_tensor(a) for a in [*s["out"], s.get("y")] if a is not None]
    elif kind == "gemv_batch":
        n, k = BITNET_2B_SHAPES[case["shape"]]
        q = torch.randint(-127, 128, (case["count"], k), generator=g, device="cuda").to(torch.int8).cpu().numpy()
        s["lib"] = kernel.load_library()
        s["keep"] = [device.DeviceArray.from_numpy(a) for a in q]
        s["xs"] = device.DeviceArray.from_numpy(rng.uniform(0.01, 0.05, 1).astype(np.float32))
        s["y"] = device.DeviceArray((case["count"], n), np.float32)
        s["args"] = (kernel.LinearArgs * case["count"])()
        for i, a in enumerate(s["args"]):
            a.w[0] = _device_weight(case["shape"], i).handle
            a.out[0] = s["y"].ptr + 4 * n * i
            a.n_mats, a.M, a.prologue, a.epilogue = 1, 1, kernel.PRO_INT8, kernel.EPI_STORE
            a.x_i8, a.x_scales = s["keep"][i].ptr, s["xs"].ptr
        s["views"] = _tensor(s["y"])
    elif kind == "host_mlp":
        s["x"] = _normal(g, case["rows"], H)
        s["gamma"], s["gamma2"] = _gamma(g, H), _gamma(g, I)
        s["w"] = [_host_weight(n) for n in ("gate", "up", "down")]
        t = case["rows"]
        s["xq"], s["hq"] = np.empty((t, H), np.int8), np.empty((t, I), np.int8)
        s["xs"], s["hs"] = np.empty(t, np.float32), np.empty(t, np.float32)
        s["tmp"] = np.empty((t, I), np.float32)
    elif kind == "decode":
        s["model"], _ = _device_model(case["family"], case["table"])
        b, ctx, steps = case["batch"], case["ctx"], case["steps"]
        s["start"] = [ctx + 11 * i for i in range(b)]      # unequal lengths
        s["state"] = runtime.init_state(s["model"], max(s["start"]) + steps + 1, batch=b, kv_dtype=case["kv"])
        for i, n in enumerate(s["start"]):
            runtime.prefill_first_token(s["state"], rng.integers(0, V, n), seq=i)
        s["tokens"] = rng.integers(0, V, (steps, b)).astype(np.int32)
    elif kind == "prefill":
        s["model"], _ = _device_model(case["family"], case["table"])
        s["state"] = runtime.init_state(s["model"], case["ctx"] + case["tokens"] + 8, kv_dtype=case["kv"])
        if case["ctx"]:
            runtime.prefill_first_token(s["state"], rng.integers(0, V, case["ctx"]))
        s["tokens"] = rng.integers(0, V, case["tokens"]).tolist()
    elif kind == "generate":
        dm, follows = _device_model("bitnet", case["table"])
        s["net"] = api.BitNet(dm, tokenizer.IdTokenizer())
        # a prompt that ends by quoting its own beginning, where prompt lookup finds the continuation
        walk = [int(rng.integers(0, V))]
        while len(walk) < case["prompt"] * 2 // 3:
            walk.append(int(follows[walk[-1]]))
        s["prompt"] = walk + walk[:case["prompt"] - len(walk)]
    else:
        dev = _keep("hybrid", _build_hybrid)
        s["state"] = _HybridState(dev, batch=case["batch"], max_steps=32)
        s["tokens"] = rng.integers(0, V, (case["prompt"], case["batch"])).astype(np.int32)
    return s


def run(s):
    kind = s["kind"]
    if kind == "linear":
        if s["block"] == "qkv":
            device.linear(s["w"], s["out"], s["rows"], x_f32=s["x"], gamma=s["gamma"], eps=EPS)
        else:
            device.linear(s["w"], s["out"], s["rows"], x_f32=s["x"], gamma=s["gamma"], eps=EPS, epilogue=kernel.EPI_RELU2_MUL)
            device.linear([s["down"]], [s["y"]], s["rows"], x_f32=s["out"][0], gamma=s["gamma2"], eps=EPS)
        return s["views"]
    if kind == "gemv_batch":
        kernel.check(s["lib"].lspk_linear_batch(s["args"], s["count"]))
        return s["views"]
    if kind == "host_mlp":
        (gate, gate_s), (up, up_s), (down, down_s) = s["w"]
        x, xq, hq = s["x"], s["xq"], s["hq"]
        if s["rows"] == 1:
            xs = kernel.rmsnorm_quantize_into(x[0], s["gamma"], xq[0], s["tmp"][0], EPS)
            g = kernel.matmul_packed_m1(xq[0], gate, gate_s, xs)
            u = kernel.matmul_packed_m1(xq[0], up, up_s, xs)
            h = kernel.relu2_mul_into(g, u, g)
            hs = kernel.rmsnorm_quantize_into(h, s["gamma2"], hq[0], s["tmp"][0], EPS)
            y = kernel.matmul_packed_m1(hq[0], down, down_s, hs)
            return h, kernel.add_inplace(y, x[0])
        kernel.rmsnorm_quantize_batched(x, s["gamma"], xq, s["xs"], s["tmp"], EPS)
        g = kernel.matmul_packed_mT(xq, s["xs"], gate, gate_s)
        u = kernel.matmul_packed_mT(xq, s["xs"], up, up_s)
        h = kernel.relu2_mul_into_batched(g, u, g)
        kernel.rmsnorm_quantize_batched(h, s["gamma2"], hq, s["hs"], s["tmp"], EPS)
        y = kernel.matmul_packed_mT(hq, s["hs"], down, down_s)
        return h, kernel.add_inplace(y.reshape(-1), x.reshape(-1)).reshape(y.shape)
    if kind == "decode":
        st, tokens = s["state"], s["tokens"]
        for i, n in enumerate(s["start"]):      # back to the end of the prompt
            st.set_pos(i, n)
        if s["logits"]:
            if s["batch"] == 1:
                return [runtime.forward_one(s["model"], st, t[0]) for t in tokens]
            return [runtime.forward_step(st, t, want_logits=True)[1] for t in tokens]
        if s["batch"] == 1:
            ids = runtime.decode_greedy(st, tokens[0, 0], s["steps"])
            return np.asarray(ids), runtime.forward_one(s["model"], st, ids[-1])
        ids = np.empty((s["steps"], s["batch"]), np.int32)
        kernel.check(st.lib.lspk_decode_greedy(st.handle, tokens[0].ctypes.data, s["steps"], ids.ctypes.data))
        return ids, runtime.forward_step(st, ids[-1], want_logits=True)[1]
    if kind == "prefill":
        st = s["state"]
        st.pos = s["ctx"]
        if s["all"]:
            return runtime.forward_prefill_all_logits(s["model"], st, s["tokens"])
        return runtime.forward_prefill(s["model"], st, s["tokens"])
    if kind == "generate":
        r = s["net"].generate(s["prompt"], s["new"], speculative=s["speculative"], return_full=True)
        return np.asarray(r.token_ids)
    st = s["state"]
    st.reset()
    first = st.prefill(s["tokens"])
    ids = st.decode_greedy(first, s["steps"])
    return first, ids, st.step(ids[-1], want_logits=True)[1]


# ---- what a pass cannot do without ----------------------------------------------------------------------------------
def _model_pass(rows, table, heads, kv_bytes, keys, new_rows):
    """Bytes and operations of `rows` token rows through the model once: every weight once, `heads` rows of logits,
    `keys` cached keys read per layer, `new_rows` of them written."""
    flops = 2.0 * LAYERS * LAYER_WEIGHTS * rows + 2.0 * V * H * heads
    b = LAYERS * LAYER_WEIGHTS / 4 + LAYERS * (3 * H + I) * 2 + (V * H * TABLE_BYTES[table] if heads else 0)
    b += LAYERS * 2 * KV * kv_bytes * (keys + new_rows) + rows * H * TABLE_BYTES[table] + 4 * V * heads
    return b, flops


def work(case):
    kind = case["kind"]
    if kind == "linear":
        m = case["rows"]
        shapes = [(H, H), (KV, H), (KV, H)] if case["block"] == "qkv" else [(I, H), (I, H), (H, I)]
        w = sum(n * k for n, k in shapes)
        rows = m * (4 * H + (4 * (H + 2 * KV) if case["block"] == "qkv" else 4 * (I + H)))
        return {"bytes": w / 4 + rows, "flops": 2.0 * m * w}
    if kind == "gemv_batch":
        n, k = BITNET_2B_SHAPES[case["shape"]]
        return {"bytes": case["count"] * (n * k / 4 + k + 4 * n), "flops": 2.0 * case["count"] * n * k}
    if kind == "host_mlp":
        m = case["rows"]
        return {"bytes": 3 * H * I / 4 + m * 4 * (H + I + H), "flops": 2.0 * m * 3 * H * I}
    if kind == "decode":
        b = case["batch"]
        kvb = 2 if case["kv"] == "fp16" else 4
        total = flops = 0.0
        steps = case["steps"] + (0 if case["logits"] or b > 1 else -1) + (0 if case["logits"] else 1)
        for t in range(steps):
            keys = sum(case["ctx"] + 11 * i + t for i in range(b))
            x, f = _model_pass(b, case["table"], b, kvb, keys, b)
            total += x
            flops += f + 4.0 * LAYERS * H * keys
        return {"bytes": total, "flops": flops}
    if kind == "prefill":
        t, ctx = case["tokens"], case["ctx"]
        b, f = _model_pass(t, case["table"], t if case["all"] else 1, 2 if case["kv"] == "fp16" else 4, ctx, t)
        return {"bytes": b, "flops": f + 4.0 * LAYERS * H * (t * ctx + t * (t + 1) / 2)}
    if kind == "generate":
        b, f = _model_pass(case["prompt"], case["table"], 1, 2, 0, case["prompt"])
        for t in range(case["new"] - 1):
            x, y = _model_pass(1, case["table"], 1, 2, case["prompt"] + t, 1)
            b, f = b + x, f + y + 4.0 * LAYERS * H * (case["prompt"] + t)
        return {"bytes": b, "flops": f}
    c, b = HYBRID, case["batch"]
    di = c.nheads * c.headdim
    mamba_w = H * (2 * di + 2 * c.d_state + c.nheads) + di * H
    expert_w = 3 * H * I
    used = c.num_experts * (1 - (1 - 2 / c.num_experts) ** b)      # experts that b rows of two choices each reach
    half = c.num_layers // 2
    states = 2 * 4 * b * (di * c.d_state + 4 * (di + 2 * c.d_state))
    step_bytes = half * (mamba_w / 4 + states + used * expert_w / 4 + c.num_experts * H * 4) + V * H * 2
    step_flops = 2.0 * b * (half * (mamba_w + 2 * expert_w) + V * H)
    steps = case["prompt"] + case["steps"] + 1
    return {"bytes": steps * step_bytes, "flops": steps * step_flops}


def tolerance(case):
    """Activations are requantised to int8 in front of every matrix: an fp32 sum that rounds differently moves single
    activations by one of 127 steps."""
    kind = case["kind"]
    if kind == "gemv_batch":
        return {"rel": 1e-6}      # the int8 rows are given: integer sums and one scale
    if kind == "generate":
        return "exact"            # token ids of a peaked distribution
    if kind == "linear" and case["block"] == "qkv":
        return {"rel": 1e-3}      # one quantiser
    if kind in ("linear", "host_mlp"):
        return {"rel": 5e-3}      # two, the second behind a squared gate
    return {"rel": 2e-2, "differ": 0.0}      # logits behind 30 layers of quantisers; greedy ids are peaked
