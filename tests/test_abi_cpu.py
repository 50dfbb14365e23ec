"""No-GPU checks of the C ABI: the shared library builds, loads, exports every symbol the header
declares, agrees with the ctypes mirror on struct sizes, and rejects bad arguments before it
touches a device."""
import ctypes as ct
import re
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def lib():
    from layer_quant_b200 import _lib, build
    build.build()
    return _lib.lib()


def declared_symbols():
    text = (ROOT / "include" / "layer_quant_b200.h").read_text()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(lq_[a-z0-9_]+)\s*\(", text)))


def test_every_declared_symbol_is_exported(lib):
    names = declared_symbols()
    assert len(names) >= 12
    for n in names:
        assert hasattr(lib, n), f"{n} declared in include/layer_quant_b200.h but not exported"


def test_struct_sizes_agree(lib):
    from layer_quant_b200 import _lib
    structs = (_lib.MxState, _lib.Rounding, _lib.MxUpdateArgs, _lib.Int4Cache, _lib.Int4DecodeArgs, _lib.DenseUpdateArgs,
               _lib.Conv1dUpdateArgs, _lib.Int4PrefillArgs)
    for which, struct in enumerate(structs):
        assert lib.lq_abi_sizeof(which) == ct.sizeof(struct), struct.__name__
    assert lib.lq_abi_sizeof(len(structs)) == -1
    assert lib.lq_abi_sizeof(99) == -1
    assert lib.lq_abi_version() == 1


def test_header_compiles_as_c(tmp_path):
    import subprocess
    src = tmp_path / "t.c"
    src.write_text('#include "layer_quant_b200.h"\nint main(void){lq_int4_decode_args a; lq_mx_update_args b; (void)a; (void)b; return 0;}\n')
    subprocess.run(["gcc", "-std=c99", "-Wall", "-Werror", "-I", str(ROOT / "include"), "-c", str(src), "-o", str(tmp_path / "t.o")], check=True)


def test_argument_validation_needs_no_device(lib):
    from layer_quant_b200 import _lib
    assert lib.lq_mx_state_update(None, None) == _lib.LQ_ERR_INVALID_ARGUMENT
    a = _lib.MxUpdateArgs()
    assert lib.lq_mx_state_update(ct.byref(a), None) == _lib.LQ_ERR_INVALID_ARGUMENT
    assert b"null state pointer" in lib.lq_last_error_string()
    a.state.q_state, a.state.shared_exp, a.state.micro_exp = 256, 512, 768
    a.state.batch, a.state.heads, a.state.dim, a.state.dstate = 1, 1, 1, 24
    a.state.format_bits = 6
    assert lib.lq_mx_state_update(ct.byref(a), None) == _lib.LQ_ERR_INVALID_ARGUMENT
    assert b"Only MX8 and MX4" in lib.lq_last_error_string()
    a.state.format_bits = 8
    assert lib.lq_mx_state_update(ct.byref(a), None) == _lib.LQ_ERR_INVALID_ARGUMENT
    assert b"divisible by 16" in lib.lq_last_error_string()
    with pytest.raises(ValueError, match="divisible by 16"):
        _lib.check(_lib.LQ_ERR_INVALID_ARGUMENT)
    d = _lib.Int4DecodeArgs()
    assert lib.lq_int4_decode_attn(ct.byref(d), None) == _lib.LQ_ERR_INVALID_ARGUMENT
    c = d.cache
    c.k_packed, c.v_packed, c.k_scale, c.v_scale = 256, 512, 768, 1024
    c.batch, c.kv_heads, c.capacity, c.head_dim, c.group_size = 1, 2, 16, 128, 48
    assert lib.lq_int4_decode_attn(ct.byref(d), None) == _lib.LQ_ERR_INVALID_ARGUMENT
    assert b"must be divisible by group_size=48" in lib.lq_last_error_string()
    c.group_size = 32
    d.q, d.out, d.q_heads, d.seq_len = 2048, 4096, 8, 17
    assert lib.lq_int4_decode_attn(ct.byref(d), None) == _lib.LQ_ERR_INVALID_ARGUMENT
    assert b"seq_len=17 outside [1, capacity=16]" in lib.lq_last_error_string()


def test_workspace_size_and_split_heuristic(lib):
    assert lib.lq_int4_decode_workspace_bytes(0, 32, 8, 128, 4) == 0
    n = lib.lq_int4_decode_workspace_bytes(2, 32, 8, 128, 4)
    assert n == 65536 * 4 + 2048 + 2 * 32 * 4 * 128 * 4
    assert lib.lq_int4_decode_auto_splits(1, 8, 1) == 1
    assert lib.lq_int4_decode_auto_splits(1, 8, 64) == 1
    s = lib.lq_int4_decode_auto_splits(1, 8, 131072)
    assert 8 <= s <= 128  # a single sequence with a long context is spread over the SMs
    assert lib.lq_int4_decode_auto_splits(256, 8, 131072) <= 4


def decode_args(batch, seq_len, gs=32, append=False, splits=0, kv_heads=8, ratio=4, dtype=None):
    """What the split count depends on (nothing here is launched: no pointer is set but the one that says whether a row is appended)."""
    from layer_quant_b200 import _lib
    a = _lib.Int4DecodeArgs()
    a.cache.batch, a.cache.kv_heads, a.cache.capacity, a.cache.head_dim, a.cache.group_size = batch, kv_heads, seq_len, 128, gs
    a.q_heads, a.seq_len, a.splits, a.dtype = ratio * kv_heads, seq_len, splits, _lib.LQ_BF16 if dtype is None else dtype
    if append:
        a.k_new = a.v_new = 256
    return a


def test_split_count_is_the_launchs_own(lib):
    """Of either kernel (group size 16: CUDA cores), on both sides of where a CTA gets all warps of an SM; given back as `splits` it stays."""
    choice = lambda *a, **k: lib.lq_int4_decode_split_count(ct.byref(decode_args(*a, **k)))
    assert choice(16, 8192, append=True) == 1 and choice(16, 8192, gs=16, append=True) == 3
    assert choice(1, 131072) == 18 and choice(18, 4000) == 1 and choice(24, 3001) == 2
    for b, n, gs in ((1, 1, 32), (1, 1024, 32), (1, 1024, 16), (3, 5000, 64), (64, 32768, 128), (200, 320, 32)):
        s = choice(b, n, gs=gs)
        assert 1 <= s <= 128 and choice(b, n, gs=gs, splits=s) == s
    for batch, tokens, s in ((48, 16383, 3), (96, 8191, 2), (16, 65535, 8), (32, 32767, 4), (64, 32767, 2)):
        assert choice(batch, tokens) == choice(batch, tokens, gs=16) == s
    assert choice(2, 130, splits=100) == 3 and choice(2, 640, splits=7) == 5 and choice(1, 131072, splits=500) == 128  # never an empty split
    assert choice(1, 1, append=True) == 1
    # fp32 queries and eight heads a kv head: CTAs of eight warps, two of four an SM, measured best or within a per cent of it at these sizes
    from layer_quant_b200 import _lib
    for kw in (dict(ratio=8), dict(ratio=8, dtype=_lib.LQ_F16), dict(dtype=_lib.LQ_F32), dict(ratio=1, dtype=_lib.LQ_F32)):
        for batch, tokens, splits in ((4, 32768, 9), (24, 12000, 3), (64, 6000, 1), (16, 8191, 1), (1, 131072, 18)):
            assert choice(batch, tokens, append=True, **kw) == splits, (batch, tokens, kw)
    assert lib.lq_int4_decode_split_count(None) == 1 and choice(0, 100) == 1 and choice(1, 0) == 1


def test_room_is_enough_for_the_choice(lib):
    """Around every length at which a tile begins, on either kernel, with and without a row appended: the choice is not monotonic in the length, and a launch
    that appends chooses for one token less."""
    for batch in (1, 2, 3, 5, 16, 18, 24, 39, 64):
        for tile in [*range(1, 100), 256, 511, 1024, 2048]:
            for n in (64 * tile - 1, 64 * tile, 64 * tile + 1, 64 * tile + 2):
                room = lib.lq_int4_decode_auto_splits(batch, 8, n)
                for gs, ratio in ((16, 4), (32, 4), (32, 8)):
                    for append in (False, True):
                        assert lib.lq_int4_decode_split_count(ct.byref(decode_args(batch, n, gs, append, ratio=ratio))) <= room, (batch, n, gs, ratio, append)
    for n in (1, 2, 2 ** 31 - 65):
        assert lib.lq_int4_decode_auto_splits(1, 8, n) >= 1


def test_no_fallback_when_library_missing(monkeypatch, tmp_path):
    from layer_quant_b200 import _lib
    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setattr(_lib, "LIB_PATH", tmp_path / "missing.so")
    with pytest.raises(RuntimeError, match="no CPU or Triton fallback"):
        _lib.lib()


def test_split_count_in_launches_around_250_us(lib):
    """Fewer splits win ties only in the longest launches (148 SMs, as on the GPU the rule was measured on and as without one)."""
    for batch, tokens, splits in ((48, 16383, 3), (96, 8191, 2), (16, 65535, 8), (32, 32767, 4), (64, 32767, 2)):
        assert lib.lq_int4_decode_auto_splits(batch, 8, tokens) == splits
