"""fp8_block_run by itself: the arguments that it refuses before any call (its place 0), and the place and code of a call that fails."""
import ctypes as C

import pytest

INVALID = 1   # cudaErrorInvalidValue
GEMM = C.CFUNCTYPE(C.c_int, C.c_int, C.c_int, C.c_int, C.c_void_p, C.c_void_p, C.c_void_p, C.c_float, C.c_void_p, C.c_void_p, C.c_int, C.c_void_p)
ADD = C.CFUNCTYPE(C.c_int, C.c_int, C.c_int, C.c_int, C.c_void_p, C.c_void_p, C.c_void_p, C.c_float, C.c_void_p, C.c_void_p, C.c_void_p)
SWIGLU = C.CFUNCTYPE(C.c_int, C.c_int, C.c_int, C.c_int, C.c_void_p, C.c_void_p, C.c_void_p, C.c_float, C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p)
FORWARD = C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_void_p, C.c_void_p)
DECODE = C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_void_p)
ENTRIES = {"gemm_scaled": GEMM, "gemm_accumulate_f32": ADD, "gemm_swiglu_raise": SWIGLU, "attention_raise": FORWARD, "attention_decode": DECODE}
B, S, H, HD, F, S_MAX = 2, 8, 2, 64, 48, 24


@pytest.fixture
def lib(built_libs):
    from goml_b200 import block_glue as BG
    lib = BG._init()
    lib.fp8_block_region_bytes.restype, lib.fp8_block_region_bytes.argtypes = C.c_size_t, [C.c_int] * 3
    lib.fp8_block_run.restype, lib.fp8_block_run.argtypes = C.c_int, [C.POINTER(BG.BlockRunArgs)]
    return lib


def block(lib, decode, pointer, entry=lambda name, *args: 0, **changed):
    """A block's arguments: buffers by pointer(name, bytes), the other libraries' calls by entry(name, *args)."""
    from goml_b200 import block_glue as BG
    seq = 1 if decode else S
    T, d = B * seq, H * HD
    region = lib.fp8_block_region_bytes(T, d, F)
    a = BG.BlockRunArgs(batch=B, seq_len=seq, d_model=d, heads=H, ffn_hidden=F, s_max=S_MAX, rope_rows=S_MAX if decode else S, decode=int(decode), eps=1e-5,
                        softmax_scale=0.1, region_bytes=region, attention_ctx=0x1000)
    a.kept = [t(lambda *args, name=name: entry(name, *args)) for name, t in ENTRIES.items()]
    for name, fn in zip(ENTRIES, a.kept):
        setattr(a, name, C.cast(fn, C.c_void_p))
    cache = B * H * S_MAX * HD
    sizes = dict(x=4 * T * d, h=4 * T * d, norm1=4 * d, norm2=4 * d, wqkv=256, wo=256, wgate_up=256, wdown=256, wqkv_scale=4, wo_scale=4, wgate_up_scale=4,
                 wdown_scale=4, cos_tab=2 * S_MAX * HD, sin_tab=2 * S_MAX * HD, k_cache=cache, v_cache=cache, cache_scales=8, cache_lens=4 * B, words=256,
                 rstd=4 * T, codes=T * d, k_codes=T * d, v_codes=T * d, region=region)
    for name, n in sizes.items():
        setattr(a, name, pointer(name, n))
    for name, value in changed.items():
        setattr(a, name, value)
    return a


ALWAYS = [{name: None} for name in (*ENTRIES, "attention_ctx", "x", "h", "wqkv", "wo", "wgate_up", "wdown", "words", "rstd", "codes", "region")]
ALWAYS += [dict(batch=0), dict(batch=-1), dict(heads=0), dict(d_model=0), dict(d_model=129), dict(ffn_hidden=0), dict(ffn_hidden=-16), dict(region_bytes=0),
           dict(region_bytes=-1), dict(v_cache=None), dict(cache_scales=None), dict(cache_lens=None)]
STEP = [dict(seq_len=2), dict(seq_len=0), dict(k_cache=None), dict(s_max=0)]
PROMPT = [dict(seq_len=0), dict(seq_len=-1), dict(batch=1 << 20, seq_len=1 << 20, rope_rows=1 << 20, s_max=1 << 20), dict(k_codes=None), dict(v_codes=None),
          dict(s_max=S - 1), dict(rope_rows=S - 1), dict(rope_rows=0)]


@pytest.mark.parametrize("decode,changed", [(decode, c) for decode in (False, True) for c in ALWAYS + (STEP if decode else PROMPT)],
                         ids=lambda v: str(v) if isinstance(v, bool) else "-".join(f"{k}={x}" for k, x in v.items()))
def test_arguments_that_are_refused(lib, decode, changed):
    # no buffer is real: a call that got as far as a kernel would return that call's place
    if changed.get("region_bytes") == -1:
        changed = dict(region_bytes=lib.fp8_block_region_bytes(B if decode else B * S, H * HD, F) - 1)
    calls = []
    assert lib.fp8_block_run(C.byref(block(lib, decode, lambda name, n: 0x10000, lambda *args: calls.append(args) or 0, norm1=0x10001, **changed))) == INVALID
    assert not calls


@pytest.mark.parametrize("decode", [False, True])
def test_the_same_arguments_unchanged_reach_the_first_call(lib, decode):
    # which refuses its misaligned weights
    for more in ({}, {} if decode else dict(k_cache=None, v_cache=None, cache_scales=None, cache_lens=None, s_max=0)):
        assert lib.fp8_block_run(C.byref(block(lib, decode, lambda name, n: 0x10000, norm1=0x10001, **more))) == 1 << 16 | INVALID
    assert lib.fp8_block_run(None) == INVALID


@pytest.mark.gpu
@pytest.mark.parametrize("decode", [False, True])
def test_place_and_code_of_a_failed_call(cuda, lib, decode):
    # the other libraries' calls are stand-ins, of which one fails; this library's own are real, and refuse a misaligned or missing
    # operand.  What stands behind a failed call is not issued
    import torch
    real = {}

    def pointer(name, n):
        real[name] = torch.zeros(n, dtype=torch.uint8, device="cuda")
        return real[name].data_ptr()

    T, d = B * (1 if decode else S), H * HD
    attention = "attention_decode" if decode else "attention_raise"
    order = [("gemm_scaled", 2), (attention, 4), ("gemm_accumulate_f32", 6), ("gemm_swiglu_raise", 8), ("gemm_accumulate_f32", 10)]
    shapes = {2: (T, 3 * d, d), 6: (T, d, d), 8: (T, F, d), 10: (T, d, F)}

    def run(fails=0, **changed):
        seen = []

        def entry(name, *args):
            expected, place = order[len(seen)]
            seen.append(place)
            assert name == expected and args[:3] == shapes.get(place, args[:3])
            return 7 if place == fails else 0

        rc = lib.fp8_block_run(C.byref(block(lib, decode, pointer, entry, **changed)))
        torch.cuda.synchronize()
        return rc, seen

    assert run() == (0, [2, 4, 6, 8, 10])
    for place in (2, 4, 6, 8, 10):
        assert run(place) == (place << 16 | 7, [p for p in (2, 4, 6, 8, 10) if p <= place])
    assert run(norm1=None) == (1 << 16 | INVALID, [])
    assert run(cos_tab=None) == (3 << 16 | INVALID, [2])
    assert run(norm2=None) == (7 << 16 | INVALID, [2, 4, 6])
    if decode:   # an odd number of values to quantise
        shapes[8], shapes[10] = (T, 20, d), (T, d, 20)
        assert run(ffn_hidden=20) == (9 << 16 | INVALID, [2, 4, 6, 8])
