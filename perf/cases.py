"""The work that a decode loop of a Nemotron-H-8B-shaped hybrid model has this package do, as timing cases.

Each case is one pass of one of five kinds, at the model's layer shapes (Mamba2: 128 heads x 64 x 128 state, 8 B/C groups,
convolution over 10240 channels; attention: 32 query / 8 kv heads of 128 dims):

    mx       one decode step's selective-state updates on an MX8 / MX4-held state, layer by layer
    attn     one decode step's attention over the packed INT4 KV cache, the new token appended
    prefill  a prompt, or a chunk of one, packed into the INT4 cache and attended over it
    handoff  the end of a prompt in the default configuration: K / V packed, SSM states quantised to MX blocks
    mixer    the unquantised decode step: convolution update and selective-state update on a floating-point state

Operands are laid out as the model's modules hand them over: x, B and C are slices of the convolution's output, dt of the
input projection's, q / k / v are transposed views of the projections, per-head parameters are expanded with stride 0.
"""
from __future__ import annotations

from types import SimpleNamespace

import torch

from layer_quant_b200 import dense_state
from layer_quant_b200 import int4_8b_attention as ia
from layer_quant_b200 import mamba_state_8b_kernel as mk

HEADS, DIM, DSTATE, GROUPS, CONV_W = 128, 64, 128, 8, 4
INNER = HEADS * DIM
CONV_DIM = INNER + 2 * GROUPS * DSTATE
PROJ_DIM = INNER + CONV_DIM + HEADS
QH, KVH, HD = 32, 8, 128
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def listed():
    return [
        # one sequence, the driver script's evaluation loop asking for the original numbers bit for bit: 24 short calls
        dict(name="mx8_b1_original_stream", kind="mx", batch=1, layers=24, bits=8, stream="reference", plan=False),
        # a small serving batch, prepared launches
        dict(name="mx8_b8", kind="mx", batch=8, layers=24, bits=8, stream="layered", plan=True),
        # a large serving batch, not a multiple of anything
        dict(name="mx8_b250", kind="mx", batch=250, layers=8, bits=8, stream="layered", plan=False),
        # a medium batch on the four-bit state
        dict(name="mx4_b64", kind="mx", batch=64, layers=24, bits=4, stream="layered", plan=False),
        # one sequence, a short context, the model's four attention layers
        dict(name="attn_b1_1024", kind="attn", batch=1, ctx=1024, layers=4, group=32, dtype="bf16", mask=False, plan=False),
        # a medium batch and context, one token short of whole tiles, prepared launches
        dict(name="attn_b16_8191", kind="attn", batch=16, ctx=8191, layers=4, group=32, dtype="bf16", mask=False, plan=True),
        # what a long-context server spends most of its time on
        dict(name="attn_b64_32768", kind="attn", batch=64, ctx=32768, layers=1, group=32, dtype="bf16", mask=False, plan=True),
        # a left-padded batch with the tokenizer's 2-D mask, half precision, the patch function's default group size
        dict(name="attn_b24_3001_masked", kind="attn", batch=24, ctx=3001, layers=4, group=64, dtype="fp16", mask=True, plan=False),
        # eight prompts from position 0
        dict(name="prefill_b8_1024", kind="prefill", batch=8, past=0, tokens=1024, group=32, dtype="bf16"),
        # the next chunk of two long prompts
        dict(name="prefill_b2_6001_2000", kind="prefill", batch=2, past=6001, tokens=2000, group=64, dtype="bf16"),
        # from prompt to decode: two attention layers and twelve Mamba2 layers, half of the model
        dict(name="handoff_b8_1024", kind="handoff", batch=8, tokens=1024, bits=8, group=64, dtype="bf16"),
        # the arm that the quantised states are compared with
        dict(name="mixer_b32_bf16", kind="mixer", batch=32, layers=24, dtype="bf16"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(lo * (hi / lo) ** rng.random())))


def draw(rng):
    kind = rng.choice(["mx"] * 4 + ["attn"] * 4 + ["prefill"] * 2 + ["handoff", "mixer"])
    if kind == "mx":
        stream = rng.choice(["layered", "layered", "layered", "reference", "deterministic"])
        batch = _log_int(rng, 1, 40 if stream == "reference" else 250)
        layers = rng.randint(8, 24) if batch <= 80 else 8  # the patch takes any subset of the Mamba2 layers
        return dict(kind=kind, batch=batch, layers=layers, bits=rng.choice([8, 8, 4]), stream=stream,
                    plan=rng.random() < 0.4)
    if kind == "attn":
        batch = _log_int(rng, 1, 200)
        ctx = _log_int(rng, 17, min(131072, 64 * 32768 // batch))
        small = batch * ctx <= 64 * 8192
        mask = small and rng.random() < 0.25
        return dict(kind=kind, batch=batch, ctx=ctx, layers=4 if small else 1, group=rng.choice([32, 32, 64, 128]),
                    dtype=rng.choice(["bf16", "bf16", "bf16", "fp16"]), mask=mask, plan=not mask and rng.random() < 0.4)
    if kind == "prefill":
        batch, tokens = _log_int(rng, 1, 12), _log_int(rng, 24, 3000)
        past = rng.choice([0, 0, _log_int(rng, 16, 8000)])
        while batch * tokens * (past + tokens / 2) > 2 * 2000 * 7000:
            batch, tokens = max(1, batch // 2), tokens * 3 // 4
        return dict(kind=kind, batch=batch, past=past, tokens=tokens, group=rng.choice([32, 64, 64, 128]),
                    dtype=rng.choice(["bf16", "bf16", "bf16", "fp16"]))
    if kind == "handoff":
        return dict(kind=kind, batch=_log_int(rng, 1, 24), tokens=_log_int(rng, 50, 2000), bits=rng.choice([8, 8, 4]),
                    group=rng.choice([32, 64, 128]), dtype=rng.choice(["bf16", "bf16", "fp32"]))
    dtype = rng.choice(["bf16", "bf16", "fp32", "fp16"])
    return dict(kind=kind, batch=_log_int(rng, 1, 20 if dtype == "fp32" else 40), layers=rng.randint(8, 24), dtype=dtype)


# ---- inputs --------------------------------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape, dtype=torch.bfloat16):
    return torch.randn(shape, generator=g, device="cuda", dtype=dtype)


def _kv(g, *shape, dtype):
    """N(0, 1) with one entry in a hundred at eight sigma: keys and values have outliers."""
    x = _randn(g, *shape, dtype=dtype)
    return torch.where(torch.rand(shape, generator=g, device="cuda", dtype=torch.float32) < 0.01, 8.0 * torch.sign(x), x)


def _ssm_params(g):
    A = -torch.exp(torch.rand(HEADS, generator=g, device="cuda") * 2.7726)
    D = torch.rand(HEADS, generator=g, device="cuda").to(torch.bfloat16)
    dt_bias = (torch.rand(HEADS, generator=g, device="cuda") * 2.0 - 4.0).to(torch.bfloat16)
    return A[:, None, None].expand(HEADS, DIM, DSTATE), D[:, None].expand(HEADS, DIM), dt_bias[:, None].expand(HEADS, DIM)


def _split_xbc(xbc):
    batch = xbc.shape[0]
    x, B, C = xbc.split([INNER, GROUPS * DSTATE, GROUPS * DSTATE], dim=-1)
    return x.reshape(batch, HEADS, DIM), B.view(batch, GROUPS, DSTATE), C.view(batch, GROUPS, DSTATE)


def _prepare_mx(case, g):
    batch, layers, bits = case["batch"], case["layers"], case["bits"]
    q = torch.empty((layers, batch, HEADS, DIM, DSTATE if bits == 8 else DSTATE // 2), device="cuda", dtype=torch.int8 if bits == 8 else torch.uint8)
    e = torch.empty((layers, batch, HEADS, DIM, DSTATE // 16), device="cuda", dtype=torch.uint8)
    m = torch.empty_like(e)
    s = SimpleNamespace(states=(q, e, m), calls=[], plans=None)
    kw = dict(dt_softplus=True, stochastic=case["stream"] != "deterministic", seed=1234,
              rng_stream=None if case["stream"] == "deterministic" else case["stream"])
    for layer in range(layers):
        first = mk.allocate_state_kernel_cache(_randn(g, batch, HEADS, DIM, DSTATE, dtype=torch.float32) * 0.5, 16, bits)
        for dst, src in ((q[layer], first.q_state), (e[layer], first.shared_exp), (m[layer], first.micro_exp)):
            dst.copy_(src)
        cache = mk.MambaStateKernelCache(q[layer], e[layer], m[layer], format_bits=bits, layout=first.layout, layer=layer)
        x, B, C = _split_xbc(_randn(g, batch, CONV_DIM))
        dt = _randn(g, batch, PROJ_DIM)[:, -HEADS:, None].expand(batch, HEADS, DIM)
        A, D, dt_bias = _ssm_params(g)
        s.calls.append((cache, (x, dt, A, B, C), dict(kw, D=D, dt_bias=dt_bias)))
    if case["plan"]:
        s.plans = [mk.MxUpdatePlan(cache, *ops, **named) for cache, ops, named in s.calls]
    return s


def _context(g, case, layer, holder, length, room):
    """A layer's cache, sized as the forward sizes it, with `length` tokens in it."""
    batch, group, dtype = case["batch"], case["group"], DTYPES[case["dtype"]]
    cache = ia._ensure_layer_cache(holder, layer, batch, KVH, room, HD, group, torch.device("cuda", torch.cuda.current_device()))
    for t in (cache.k_packed, cache.v_packed, cache.k_scale, cache.v_scale):
        t.zero_()
    step = max(1, (1 << 26) // (batch * KVH * HD))
    for at in range(0, length, step):
        n = min(step, length - at)
        k, v = (_kv(g, batch, KVH, n, HD, dtype=dtype) for _ in range(2))
        ia._pack_kv_into_cache(cache, k, v, torch.arange(at, at + n, device="cuda"), group, known_len=at + n)
    return cache


def _heads(t, n):
    return t.view(t.shape[0], t.shape[1], n, HD).transpose(1, 2)


def _prepare_attn(case, g):
    batch, ctx, group, dtype = case["batch"], case["ctx"], case["group"], DTYPES[case["dtype"]]
    s = SimpleNamespace(calls=[], plans=None, mask=None)
    if case["mask"]:  # left padding: each sequence starts somewhere in the first half
        start = torch.randint(0, max(1, ctx // 2), (batch, 1), generator=g, device="cuda")
        s.mask = (torch.arange(ctx, device="cuda")[None] >= start).to(torch.int64)
    holder = SimpleNamespace()
    for layer in range(case["layers"]):
        cache = _context(g, case, layer, holder, ctx - 1, ctx)
        q = _heads(_randn(g, batch, 1, QH * HD, dtype=dtype), QH)
        k, v = (_heads(_kv(g, batch, 1, KVH * HD, dtype=dtype), KVH) for _ in range(2))
        s.calls.append((q, k, v, cache))
    if case["plan"]:
        s.plans = [ia.Int4DecodePlan(q, cache, ctx, group, k_new=k, v_new=v) for q, k, v, cache in s.calls]
    return s


def _prepare_prefill(case, g):
    batch, past, tokens, dtype = case["batch"], case["past"], case["tokens"], DTYPES[case["dtype"]]
    cache = _context(g, case, 0, SimpleNamespace(), past, past + tokens)
    q = _heads(_randn(g, batch, tokens, QH * HD, dtype=dtype), QH)
    k, v = (_heads(_kv(g, batch, tokens, KVH * HD, dtype=dtype), KVH) for _ in range(2))
    return SimpleNamespace(q=q, k=k, v=v, cache=cache, positions=torch.arange(past, past + tokens, device="cuda"))


def _prepare_handoff(case, g):
    batch, tokens, dtype = case["batch"], case["tokens"], DTYPES[case["dtype"]]
    holder, s = SimpleNamespace(), SimpleNamespace(kv=[], states=[], positions=torch.arange(tokens, device="cuda"))
    for layer in range(2):
        k, v = (_heads(_kv(g, batch, tokens, KVH * HD, dtype=dtype), KVH) for _ in range(2))
        s.kv.append((_context(g, case, layer, holder, 0, tokens), k, v))
    for layer in range(12):
        s.states.append(_randn(g, batch, HEADS, DIM, DSTATE, dtype=dtype) * 0.5)
    return s


def _prepare_mixer(case, g):
    batch, layers, dtype = case["batch"], case["layers"], DTYPES[case["dtype"]]
    s = SimpleNamespace(conv=_randn(g, layers, batch, CONV_DIM, CONV_W), ssm=torch.empty((layers, batch, HEADS, DIM, DSTATE), device="cuda", dtype=dtype), calls=[])
    for layer in range(layers):
        s.ssm[layer] = _randn(g, batch, HEADS, DIM, DSTATE, dtype=dtype) * 0.5
        proj = _randn(g, batch, PROJ_DIM)
        _, xbc, dt = proj.split([INNER, CONV_DIM, HEADS], dim=-1)
        weight, bias = _randn(g, CONV_DIM, CONV_W) * 0.5, _randn(g, CONV_DIM) * 0.1
        A, D, dt_bias = _ssm_params(g)
        s.calls.append((xbc, s.conv[layer], weight, bias, s.ssm[layer], dt[:, :, None].expand(-1, -1, DIM), A, D, dt_bias))
    return s


def prepare(case, seed):
    g = _gen(seed)
    s = {"mx": _prepare_mx, "attn": _prepare_attn, "prefill": _prepare_prefill, "handoff": _prepare_handoff, "mixer": _prepare_mixer}[case["kind"]](case, g)
    s.case = case
    return s


# ---- one pass ------------------------------------------------------------------------------------------------------

def _cache_tensors(cache):
    return cache.k_packed, cache.v_packed, cache.k_scale, cache.v_scale


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "mx":
        if s.plans is not None:
            y = [plan.run() for plan in s.plans]
        else:
            y = [mk.mx_state_selective_update(cache, *ops, **named) for cache, ops, named in s.calls]
        return y, s.states
    if kind == "attn":
        if s.plans is not None:
            out = [plan.launch() for plan in s.plans]
        else:
            out = [ia._append_decode_attention(q, k, v, cache, case["ctx"], QH // KVH, case["group"], attention_mask=s.mask)
                   for q, k, v, cache in s.calls]
        return out, [_cache_tensors(c[3]) for c in s.calls]
    if kind == "prefill":
        ia._pack_kv_into_cache(s.cache, s.k, s.v, s.positions, case["group"], known_len=case["past"] + case["tokens"])
        out = ia._prefill_attention(s.q, s.cache, QH // KVH, case["group"], first_len=case["past"] + 1)
        return out, _cache_tensors(s.cache)
    if kind == "handoff":
        for cache, k, v in s.kv:
            ia._pack_kv_into_cache(cache, k, v, s.positions, case["group"], known_len=case["tokens"])
        mx = [mk.allocate_state_kernel_cache(state, 16, case["bits"]) for state in s.states]
        return [_cache_tensors(c) for c, _, _ in s.kv], [(c.q_state, c.shared_exp, c.micro_exp) for c in mx]
    y = []
    for xbc, conv_state, weight, bias, state, dt, A, D, dt_bias in s.calls:
        x, B, C = _split_xbc(dense_state.causal_conv1d_update(xbc, conv_state, weight, bias, "silu"))
        y.append(dense_state.selective_state_update(state, x, dt, A, B, C, D=D, dt_bias=dt_bias, dt_softplus=True))
    return y, s.conv, s.ssm


# ---- what a pass cannot do without ---------------------------------------------------------------------------------

def work(case):
    kind, batch = case["kind"], case["batch"]
    size = 4 if case.get("dtype") == "fp32" else 2
    values = batch * HEADS * DIM * DSTATE
    small = batch * (2 * INNER + HEADS + 2 * GROUPS * DSTATE) * 2  # x, y, dt, B, C of one layer
    if kind == "mx":
        block = 18 if case["bits"] == 8 else 10
        return {"bytes": case["layers"] * (2 * values // 16 * block + small), "flops": case["layers"] * 5 * values}
    if kind == "mixer":
        conv = batch * CONV_DIM * (2 * CONV_W + 2) * 2 + CONV_DIM * (CONV_W + 1) * 2
        return {"bytes": case["layers"] * (2 * values * size + small + conv), "flops": case["layers"] * (5 * values + 2 * batch * CONV_DIM * CONV_W)}
    row = HD + 2 * 4 * (HD // case["group"])  # K and V codes and scales of one token of one kv head
    if kind == "attn":
        ctx = case["ctx"]
        one = batch * (KVH * ctx * row + 2 * KVH * HD * size + 2 * QH * HD * size)
        return {"bytes": case["layers"] * one + (batch * ctx * 8 if case["mask"] else 0), "flops": case["layers"] * 4 * batch * QH * HD * ctx}
    tokens = case["tokens"]
    pack = batch * KVH * tokens * (2 * HD * size + row)
    if kind == "handoff":
        return {"bytes": 2 * pack + 12 * (values * size + values // 16 * (18 if case["bits"] == 8 else 10)), "flops": 0}
    seen = tokens * case["past"] + tokens * (tokens + 1) // 2  # (query, key) pairs of one head
    return {"bytes": pack + batch * KVH * case["past"] * row + 2 * batch * QH * tokens * HD * size, "flops": 4 * batch * QH * HD * seen}


def tolerance(case):
    if case["kind"] == "handoff":  # codecs: IEEE division, round half even
        return "exact"
    if case["kind"] == "mx":
        # y is bf16; a state code sits next to a rounding edge once in a few thousand, where the last bit of exp() decides
        return {"rel": 5e-3, "differ": 1e-3}
    # outputs in a 16-bit type from fp32 sums; codes, scales and everything stored in the cache follow exactly
    return {"rel": 2e-3 if case.get("dtype") == "fp16" else 5e-3}
