"""fp8_block_run by itself: the arguments that it refuses before any call (its place 0), and the place and code of a call that fails."""
import ctypes as C

import pytest

INVALID, NOT_SUPPORTED = 1, 801   # cudaErrorInvalidValue, cudaErrorNotSupported
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


def run_rows(lib, args, rows):
    """fp8_block_run_rows with rows(argument block) in fp8_gemm_rows' place (the same function object has other types elsewhere)."""
    from goml_b200 import fp8_gemm as G
    kind = C.CFUNCTYPE(C.c_int, C.POINTER(G.RowsArgs))
    keep = kind(lambda block: rows(block.contents))
    fn = lib["fp8_block_run_rows"]
    fn.restype, fn.argtypes = C.c_int, [C.c_void_p, C.c_void_p]
    return fn(C.addressof(args), C.cast(keep, C.c_void_p))


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


def test_a_step_whose_first_product_takes_rows(lib):
    # it is the first call, and its failure the end; a prompt has no such products; the arguments are refused as without them
    seen = []
    refuse = lambda g: seen.append(g.source) or 7
    assert run_rows(lib, block(lib, True, lambda name, n: 0x10000, norm1=0x10001), refuse) == 11 << 16 | 7 and seen == [1]
    assert run_rows(lib, block(lib, False, lambda name, n: 0x10000, norm1=0x10001), refuse) == 1 << 16 | INVALID and seen == [1]
    assert run_rows(lib, block(lib, True, lambda name, n: 0x10000, norm1=0x10001), lambda g: NOT_SUPPORTED) == 1 << 16 | INVALID
    for changed in (dict(seq_len=2), dict(k_cache=None), dict(x=None), dict(region_bytes=0)):
        assert run_rows(lib, block(lib, True, lambda name, n: 0x10000, **changed), refuse) == INVALID and seen == [1]


@pytest.mark.parametrize("batch,heads,taken", [(1, 64, True), (2, 64, True), (4, 32, True), (1, 65, True), (2, 65, False), (3, 64, False), (64, 2, True), (65, 2, False),
                                               (1, 128, True), (1, 130, False)])
def test_long_rows_have_a_quantiser_ahead(lib, batch, heads, taken):
    # past 8192 values the maximum that every thread block takes for itself costs more than a kernel that takes it once
    d, seen = heads * HD, []
    args = block(lib, True, lambda name, n: 0x10000, norm1=0x10001, batch=batch, heads=heads, d_model=d, region_bytes=lib.fp8_block_region_bytes(batch, d, F))
    assert run_rows(lib, args, lambda g: seen.append((g.m, g.k)) or 7) == (11 << 16 | 7 if taken else 1 << 16 | INVALID)
    assert seen == ([(batch, d)] if taken else []) and taken == (batch * d <= 8192)


@pytest.mark.gpu
@pytest.mark.parametrize("refused", [(), (11,), (12,), (13,), (14,), (11, 12), (11, 13), (12, 14), (11, 12, 13, 14)], ids=lambda r: "-".join(map(str, r)) or "none")
def test_products_that_take_rows_and_those_that_do_not(cuda, lib, refused):
    # each product by itself goes the one way or the other: which calls are made in which order, what they are given, and that the
    # stream is in h where the product behind adds to it in place
    import torch
    d, real, g = H * HD, {}, torch.Generator(device="cuda").manual_seed(1)

    def pointer(name, n):
        real[name] = torch.zeros(n, dtype=torch.uint8, device="cuda")
        return real[name].data_ptr()

    def run(fails=0):
        seen, blocks = [], {}

        def entry(name, *args):
            seen.append({"gemm_scaled": 2, "attention_decode": 4, "gemm_swiglu_raise": 8}.get(name) or (6 if args[2] == d else 10))
            return 0

        def rows(g):
            place = 11 + len(blocks)
            blocks[place] = {name: getattr(g, name) for name, _ in g._fields_}
            if place in refused and place != fails:
                return NOT_SUPPORTED
            seen.append(place)
            return 7 if place == fails else 0

        args = block(lib, True, pointer, entry)
        real["x"].copy_(torch.randn(B * d, generator=g, device="cuda").view(torch.uint8))
        rc = run_rows(lib, args, rows)
        torch.cuda.synchronize()
        return rc, seen, blocks, args

    order = [2 if 11 in refused else 11, 4, 6 if 12 in refused else 12, 8 if 13 in refused else 13, 10 if 14 in refused else 14]
    rc, seen, got, a = run()
    assert rc == 0 and seen == order
    in_place = 11 in refused or 12 in refused   # the norm or a copy brings x to h; else the second product reads x itself
    assert torch.equal(real["h"], real["x"] if in_place else torch.zeros_like(real["h"]))
    hidden = a.words + 4 * 6   # the maximum of the hidden activations, the last of the seven words that the first kernel clears
    none = dict(gamma=None, amax=None, c=None, x=None, x_in=None, h=None, h_amax=None, zero=None, zeros=0, b_complete=1, reserved=0)
    common = lambda w, **more: {**none, "b": getattr(a, w), "scale_b": getattr(a, w + "_scale"), "m": B, "stream": a.stream, "eps": pytest.approx(1e-5), **more}
    assert got[11] == common("wqkv", source=1, rows=a.x, gamma=a.norm1, c=got[11]["c"], n=3 * d, k=d, zero=a.words, zeros=7, b_complete=0)
    assert got[12] == common("wo", source=2, rows=got[12]["rows"], x=a.h, x_in=a.h if 11 in refused else a.x, n=d, k=d)
    assert got[13] == common("wgate_up", source=1, rows=a.h, gamma=a.norm2, h=got[13]["h"], h_amax=hidden, n=F, k=d)
    assert got[14] == common("wdown", source=3, rows=got[13]["h"], amax=hidden, x=a.h, x_in=a.h, n=d, k=F)
    inside = lambda p: a.region <= p < a.region + a.region_bytes and p % 16 == 0
    assert inside(got[11]["c"]) and inside(got[12]["rows"]) and inside(got[13]["h"])
    assert real["cache_lens"].view(torch.int32).tolist() == [1] * B
    for place in (11, 12, 13, 14):
        if place not in refused:
            assert run(place)[:2] == (place << 16 | 7, order[:order.index(place) + 1])
