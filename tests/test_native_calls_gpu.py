"""The C++ call path of the host mirrors against the general path through ctypes: the same launch, so the same bits."""
import pytest
import torch

from tests.util import dev

pytestmark = pytest.mark.gpu


def _cache(m, b, hkv, tlen, gs, g):
    cache = m._allocate_layer_cache(b, hkv, 256, 128, 128 // gs, dev())
    k, v = (torch.randn(b, hkv, tlen, 128, generator=g, device=dev()) for _ in range(2))
    m._pack_kv_into_cache(cache, k, v, torch.arange(tlen, device=dev()), gs)
    return cache


@pytest.mark.parametrize("kind", ["bool", "uint8", "int32", "int64", "int64_wide", "bool4", "f32_4", "bf16_4", "f16_4", "f32_4_one", "f32_2"])
def test_masks_are_read_in_their_own_type(kind):
    """Every mask the kernel reads directly equals the fp32 bias that the host conversion makes of it."""
    from layer_quant_b200 import int4_8b_attention as m
    g = torch.Generator(device=dev()).manual_seed(3)
    b, tlen, gs = 3, 130, 32
    cache = _cache(m, b, 2, tlen, gs, g)
    q = torch.randn(b, 8, 1, 128, generator=g, device=dev()).to(torch.bfloat16)
    keep = torch.rand(b, tlen + 7, generator=g, device=dev()) < 0.7
    keep[:, -1] = True
    bias = torch.randn(b, 1, 2, tlen + 7, generator=g, device=dev())
    mask = {"bool": keep[:, :tlen], "uint8": keep[:, :tlen].to(torch.uint8), "int32": keep[:, :tlen].int(), "int64": keep[:, :tlen].long(),
            "int64_wide": keep.long(), "bool4": keep[:, None, None, :], "f32_4": bias, "bf16_4": bias.bfloat16(), "f16_4": bias.half(),
            "f32_4_one": bias[:1], "f32_2": keep.float()}[kind]
    out = m._decode_attention(q, cache, tlen, 4, gs, attention_mask=mask)
    general = m._launch_decode(q, cache, tlen, gs, m._decode_attention_mask(mask, b, tlen, dev()))
    assert torch.equal(out, general)


@pytest.mark.parametrize("case", ["plain", "z", "given_out", "step_counter", "no_D", "fp32_operands", "half_up", "layered4", "reference_layout"])
def test_state_update_equals_the_prepared_call(case):
    from layer_quant_b200 import mamba_state_8b_kernel as m
    g = torch.Generator(device=dev()).manual_seed(5)
    b, h, p, n, grp = 2, 4, 16, 128, 2
    dtype = torch.float32 if case == "fp32_operands" else torch.bfloat16
    r = lambda *s: torch.randn(*s, generator=g, device=dev()).to(dtype)
    state = torch.randn(b, h, p, n, generator=g, device=dev())
    x, dt, B, C = r(b, h, p), r(b, h)[:, :, None].expand(b, h, p), r(b, grp, n), r(b, grp, n)
    A = -torch.rand(h, generator=g, device=dev())[:, None, None].expand(h, p, n)
    D, bias = (None if case == "no_D" else r(h)[:, None].expand(h, p)), r(h)[:, None].expand(h, p)
    kw = dict(D=D, z=r(b, h, p) if case == "z" else None, dt_bias=bias, dt_softplus=True, stochastic=case != "half_up", seed=2**63 + 5,
              rng_stream="layered4" if case == "layered4" else "layered")
    ys, caches = [], []
    for prepared in (False, True):
        cache = m.allocate_state_kernel_cache(state, layout="reference" if case == "reference_layout" else "packed")
        cache.step, cache.layer = 7, 3
        if case == "step_counter":
            cache.step_counter = torch.full((1,), 2, dtype=torch.int64, device=dev())
        out = torch.empty_like(x) if case == "given_out" else None
        if prepared:
            y = m.MxUpdatePlan(cache, x, dt, A, B, C, out=out, step_counter=cache.step_counter, **kw).run()
        else:
            y = m.mx_state_selective_update(cache, x, dt, A, B, C, out=out, **kw)
            assert out is None or y is out
            assert cache.step == (7 if case == "step_counter" else 8)
            assert case != "step_counter" or cache.step_counter.item() == 3
        ys.append(y)
        caches.append(cache)
    assert torch.equal(*ys)
    for name in ("q_state", "shared_exp", "micro_exp"):
        assert torch.equal(getattr(caches[0], name), getattr(caches[1], name))


def test_errors_come_from_the_general_path():
    from layer_quant_b200 import dense_state, int4_8b_attention as ia, mamba_state_8b_kernel as mk
    d = dev()
    cache = mk.allocate_state_kernel_cache(torch.zeros(1, 2, 16, 128, device=d))
    x, A, B = torch.zeros(1, 2, 8, device=d), torch.zeros(2, 16, 128, device=d), torch.zeros(1, 1, 128, device=d)
    with pytest.raises(ValueError, match="Expected x shape"):
        mk.mx_state_selective_update(cache, x, x, A, B, B)
    x = torch.zeros(1, 2, 16, device=d)
    with pytest.raises(ValueError, match="unknown rng_stream"):
        mk.mx_state_selective_update(cache, x, x, A, B, B, rng_stream="other")
    for option in ("dt_softplus", "stochastic"):  # an option without a truth value
        with pytest.raises(RuntimeError, match="ambiguous"):
            mk.mx_state_selective_update(cache, x, x, A, B, B, **{option: torch.ones(2)})
    with pytest.raises(RuntimeError, match="ambiguous"):
        dense_state.selective_state_update(torch.zeros(1, 2, 16, 128, device=d), x, x, A, B, B, dt_softplus=torch.ones(2))
    for shape in ((1, 2, 8), (1, 1, 16), (2, 2, 16), (2, 16)):  # the kernel would write with these strides
        with pytest.raises(ValueError, match="Expected out shape"):
            mk.mx_state_selective_update(cache, x, x, A, B, B, out=torch.zeros(shape, device=d))
        with pytest.raises(ValueError, match="Expected out shape"):
            mk.MxUpdatePlan(cache, x, x, A, B, B, out=torch.zeros(shape, device=d))
    assert cache.step == 0
    kv = ia._allocate_layer_cache(1, 2, 16, 128, 4, torch.device(d))
    q = torch.zeros(1, 8, 1, 128, device=d, dtype=torch.bfloat16)
    with pytest.raises(ValueError, match="outside"):
        ia._decode_attention(q, kv, 17, 4, 32)
    for groups in (2, 0, -1):
        with pytest.raises(ValueError, match="query heads"):
            ia._decode_attention(q, kv, 4, groups, 32)
    with pytest.raises(ValueError, match="only supports 2D or 4D"):
        ia._decode_attention(q, kv, 4, 4, 32, attention_mask=torch.zeros(1, 1, 4, device=d))
    with pytest.raises(ValueError, match="do not match state"):
        dense_state.selective_state_update(torch.zeros(1, 2, 16, 128, device=d), x[:, :, :8], x, A, B, B)


def test_recorded_decode_owns_its_scratch():
    """A recorded decode call whose splits need scratch replays correctly whatever eager calls do to the scratch of its stream: grow it, or
    push it out with calls on more streams than are kept; the memory they gave back is filled with ones (tickets that start there never
    come to their end, and the output is not written)."""
    from layer_quant_b200 import int4_8b_attention as m
    g = torch.Generator(device=dev()).manual_seed(9)
    tlen, gs, splits = 250, 32, 4
    small, large = (_cache(m, b, 2, tlen, gs, g) for b in (2, 64))
    q = torch.randn(2, 8, 1, 128, generator=g, device=dev()).to(torch.bfloat16)
    q_large = torch.randn(64, 8, 1, 128, generator=g, device=dev()).to(torch.bfloat16)
    want = m._decode_attention(q, small, tlen, 4, gs, splits=splits)
    want_large = m._decode_attention(q_large, large, tlen, 4, gs, splits=splits)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        m._decode_attention(q, small, tlen, 4, gs, splits=splits)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        first = m._decode_attention(q, small, tlen, 4, gs, splits=splits)
        second = m._decode_attention(q_large, large, tlen, 4, gs, splits=splits)  # larger: the capture's scratch grows, too
        third = m._decode_attention(q, small, tlen, 4, gs, splits=splits)

    def check():
        for out in (first, second, third):
            out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(first, want) and torch.equal(third, want) and torch.equal(second, want_large)

    check()
    with torch.cuda.stream(stream):
        assert torch.equal(m._decode_attention(q_large, large, tlen, 4, gs, splits=splits), want_large)
        held = [torch.full((1 << 20,), 1, dtype=torch.uint8, device=dev()) for _ in range(64)]
    check()
    streams = {s.cuda_stream: s for p in (0, -1, -2, -3) for s in (torch.cuda.Stream(priority=p) for _ in range(32))}
    assert len(streams) > 64
    for s in streams.values():
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            assert torch.equal(m._decode_attention(q, small, tlen, 4, gs, splits=splits), want)
    with torch.cuda.stream(stream):
        held += [torch.full((1 << 20,), 1, dtype=torch.uint8, device=dev()) for _ in range(64)]
    check()
    assert held


def test_split_count_is_chosen_once(tmp_path):
    """A call asks for the library's choice once and launches with it; a prepared launch has asked when it was made."""
    import ctypes
    import subprocess
    from pathlib import Path
    from layer_quant_b200 import _lib
    from layer_quant_b200 import int4_8b_attention as m
    include = Path(_lib.__file__).resolve().parents[1] / "include"
    names = ("mx_state_update", "mx_quantize", "counter_add", "int4_kv_append", "int4_decode_auto_splits", "int4_prefill_attn",
             "dense_state_update", "causal_conv1d_update")
    source = tmp_path / "counts.c"
    source.write_text('#include "layer_quant_b200.h"\nint asked, launched;\n' + "".join(f"int stand_in_{n}(void) __asm__(\"lq_{n}\");\nint stand_in_{n}(void) {{ return 0; }}\n" for n in names) +
                      "int32_t lq_int4_decode_split_count(const lq_int4_decode_args* a) { asked += 1; return a->splits ? -1 : 3; }\n"
                      "size_t lq_int4_decode_workspace_bytes(int32_t b, int32_t q, int32_t k, int32_t d, int32_t s) { return s == 3 ? 4096 : 0; }\n"
                      "int lq_int4_decode_attn(const lq_int4_decode_args* a, void* s) { launched = a->workspace_bytes >= 4096 ? a->splits : -1; return 0; }\n")
    subprocess.run(["gcc", "-shared", "-fPIC", "-I", str(include), str(source), "-o", str(tmp_path / "counts.so")], check=True)
    cache = m._allocate_layer_cache(2, 2, 256, 128, 4, dev())
    q = torch.zeros(2, 8, 1, 128, dtype=torch.bfloat16, device=dev())
    native, counts = _lib.native(), ctypes.CDLL(str(tmp_path / "counts.so"))
    asked, launched = (ctypes.c_int.in_dll(counts, n) for n in ("asked", "launched"))
    native.bind(str(tmp_path / "counts.so"))
    try:
        m._decode_attention(q, cache, 200, 4, 32)
        assert (asked.value, launched.value) == (1, 3)
        plan = m.Int4DecodePlan(q, cache, 200, 32)
        assert plan.args.splits == _lib.lib().lq_int4_decode_split_count(ctypes.byref(plan.args)) >= 1
        plan.launch()
        assert asked.value == 1
    finally:
        native.bind(str(_lib.LIB_PATH))


def test_other_threads_run_during_a_launch(tmp_path):
    """A launch blocks while CUDA's queue is full.  Here a stand-in for the library blocks in every call; another thread keeps running."""
    import ctypes
    import subprocess
    import threading
    import time
    from layer_quant_b200 import _lib
    names = ("mx_state_update", "mx_quantize", "counter_add", "int4_kv_append", "int4_decode_attn", "int4_decode_workspace_bytes",
             "int4_decode_auto_splits", "int4_prefill_attn", "dense_state_update", "causal_conv1d_update")
    source = tmp_path / "slow.c"
    source.write_text("int usleep(unsigned);\n" + "".join(f"int lq_{n}(void) {{ usleep(400000); return 0; }}\n" for n in names))
    subprocess.run(["gcc", "-shared", "-fPIC", str(source), "-o", str(tmp_path / "slow.so")], check=True)
    native, block = _lib.native(), ctypes.create_string_buffer(4096)
    address, index = ctypes.addressof(block), dev().index
    native.bind(str(tmp_path / "slow.so"))
    try:
        for call in (lambda: native.mx_plan_run(address, index, 0), lambda: native.int4_plan_launch(address, index)):
            thread = threading.Thread(target=call)
            longest, last = 0.0, time.perf_counter()
            thread.start()
            while thread.is_alive():
                time.sleep(0.001)
                now = time.perf_counter()
                longest, last = max(longest, now - last), now
            assert longest < 0.2
    finally:
        native.bind(str(_lib.LIB_PATH))
