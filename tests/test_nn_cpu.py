"""What the decoder block takes and refuses before it launches anything: on the CPU."""
import pytest
import torch

from goml_b200 import nn

B, H, S_MAX, HD = 2, 4, 24, 64
CPU = torch.device("cpu")


def cache(**replaced):
    c = nn.FP8KVCache(B, H, S_MAX, HD, device="cpu")
    for name, t in replaced.items():
        setattr(c, name, t)
    return c


def block():
    blk = nn.FP8DecoderBlock.__new__(nn.FP8DecoderBlock)   # no weights: nothing here gets as far as a kernel
    blk.d, blk.H, blk.hd, blk.F = H * HD, H, HD, 128
    return blk


u8 = lambda *shape, **kw: torch.zeros(shape, dtype=torch.uint8, **kw)
BAD_CACHES = {
    "another device": lambda: cache(k=u8(B, H, S_MAX, HD, device="meta")),
    "lengths on another device": lambda: cache(lens=torch.zeros(B, dtype=torch.int32, device="meta")),
    "scales on another device": lambda: cache(scales=torch.ones(2, device="meta")),
    "rows of a longer cache": lambda: cache(v=u8(B, H, S_MAX + 1, HD)[:, :, :S_MAX]),
    "another capacity": lambda: cache(k=u8(B, H, S_MAX + 1, HD)),
    "heads and rows swapped": lambda: cache(k=u8(B, S_MAX, H, HD).transpose(1, 2)),
    "too few sequences": lambda: cache(k=u8(B - 1, H, S_MAX, HD)),
    "two bytes a code": lambda: cache(k=torch.zeros(B, H, S_MAX, HD, dtype=torch.float16)),
    "long lengths": lambda: cache(lens=torch.zeros(B, dtype=torch.int64)),
    "lengths with gaps": lambda: cache(lens=torch.zeros(2 * B, dtype=torch.int32)[::2]),
}


@pytest.mark.parametrize("name", BAD_CACHES)
def test_caches_that_kernels_cannot_be_given(name):
    bad = BAD_CACHES[name]()
    assert not bad.takes(B, H, 8, HD, CPU) and not bad.dense_on(CPU)
    with pytest.raises(ValueError, match="decode_step"):
        block().decode_step(torch.zeros(B, H * HD), bad)


def test_caches_that_they_can():
    c = cache()
    assert c.dense_on(CPU) and c.takes(B, H, S_MAX, HD, CPU)
    assert not c.takes(B, H, S_MAX + 1, HD, CPU) and not c.takes(B + 1, H, 8, HD, CPU)
    assert not c.takes(B, H, 8, HD, torch.device("cuda", 1)) and not c.dense_on(torch.device("cuda", 1))
    # what a step reads through its pointer, and a prompt is copied into
    for other in (dict(k=u8(B, H, S_MAX, HD).view(torch.float8_e4m3fn)), dict(lens=torch.zeros(B + 1, dtype=torch.int32))):
        assert cache(**other).dense_on(CPU) and not cache(**other).takes(B, H, 8, HD, CPU)


T, D = 6, 32


def rows_of(n, d, offset=0):
    room = torch.zeros(n * d + 64)
    start = -room.data_ptr() // 4 % 8 + offset      # 32-byte aligned, and `offset` values past that
    x = room[start:start + n * d].view(n, d)
    x.copy_(torch.arange(n * d, dtype=torch.float32).view(n, d))
    return x


INPUTS = {   # the input, and whether the first kernel can read it where it is
    "dense": (lambda: rows_of(T, D), True),
    "misaligned": (lambda: rows_of(T, D, 1), False),
    "rows of a wider tensor": (lambda: rows_of(T, 2 * D)[:, :D], False),
    "every other row": (lambda: rows_of(2 * T, D)[::2], False),
    "one row for all": (lambda: rows_of(1, D).expand(T, D), False),
    "bf16": (lambda: rows_of(T, D).bfloat16(), False),
    "double": (lambda: rows_of(T, D).double(), False),
    "needs a gradient": (lambda: rows_of(T, D).requires_grad_(), False),
}


@pytest.mark.parametrize("name", INPUTS)
def test_the_streams_start(name):
    make, direct = INPUTS[name]
    x = make()
    src, h = nn._stream_start(x, T, D)
    assert (src is x) == direct and (src is h) != direct
    assert h.shape == (T, D) and h.is_contiguous() and h.dtype == torch.float32 and h.data_ptr() != x.data_ptr()
    assert torch.equal(src, x.float())


@pytest.mark.parametrize("name,x", [("columns", rows_of(D, T).t()), ("sequences behind one another", rows_of(T, D).view(3, 2, D).transpose(0, 1)),
                                    ("three dimensions", rows_of(T, D).view(2, 3, D)), ("a row too few", rows_of(T - 1, D)),
                                    ("a row too many", rows_of(T + 1, D)), ("shorter rows", rows_of(2 * T, D // 2))])
def test_inputs_that_are_no_rows_are_refused(name, x):
    with pytest.raises(AssertionError):
        nn._stream_start(x, T, D)


def test_a_cache_with_a_fill_of_its_own_has_it_called():
    class Counting(nn.FP8KVCache):
        def fill(self, *args):
            super().fill(*args)

    class Duck:   # anything with a fill was good enough for the prompt
        def fill(self, k_codes, v_codes, scales, S):
            pass

    patched = cache()
    patched.fill = lambda *args: None
    assert nn._writes_directly(cache(), B, H, 8, HD, CPU)
    for c in (Counting(B, H, S_MAX, HD, device="cpu"), Duck(), patched, None):
        assert not nn._writes_directly(c, B, H, 8, HD, CPU)


def test_a_layer_with_a_product_of_its_own_has_it_called(monkeypatch):
    # for every kind of tensor, the one that goes straight to the libraries too
    from goml_b200 import fp8_gemm as G, quantize as Q
    calls = []
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: type("Stream", (), {"cuda_stream": 7}))
    monkeypatch.setattr(Q, "QuantizeF32ToF8E4M3", lambda src, dst, scale, amax, n, stream: calls.append(("quantise", n, stream)))
    monkeypatch.setattr(G, "FP8GEMMScaled", lambda m, n, k, *args: calls.append(("product", m, n, k)))

    class OnGPU(torch.Tensor):
        is_cuda = property(lambda self: True)

    class Other(nn.FP8Linear):
        def forward_codes(self, xq, M):
            assert isinstance(xq, nn.FP8Tensor) and xq.codes.shape == (M, 32)
            return "its own"

    def layer(cls):
        made = cls.__new__(cls)
        made.out_features, made.in_features, made.w = 5, 32, nn.FP8Tensor(u8(5, 32), torch.ones(2))
        return made

    x = torch.ones(3, 2, 32).as_subclass(OnGPU)
    for same in (x, x.bfloat16(), torch.ones(3, 2, 64).as_subclass(OnGPU)[..., ::2]):
        assert layer(nn.FP8Linear)(same).shape == (6, 5) and calls == [("quantise", 6 * 32, 7), ("product", 6, 5, 32)]
        patched = layer(nn.FP8Linear)
        patched.forward_codes = lambda xq, M: ("patched", M)
        assert layer(Other)(same) == "its own" and patched(same) == ("patched", 6)
        calls.clear()


# the calls of a block in their order, and what their bindings raise
CALLS = ["fp8_rmsnorm_quantize_into", "fp8_gemm_scaled", None, None, "fp8_permute_quantize_heads", "fp8_gemm_accumulate_f32", "fp8_rmsnorm_quantize_into",
         "fp8_gemm_swiglu_raise", "fp8_quantize_bf16", "fp8_gemm_accumulate_f32"]


@pytest.mark.parametrize("kind", ["step", "prompt", "prompt into a cache"])
def test_a_failed_call_is_named(monkeypatch, kind):
    from goml_b200 import block_glue as BG, fa_forward as F, fp8_gemm as G
    calls = list(CALLS)
    calls[2:4] = {"step": ["fp8_decode_rope_append", "fa_decode"], "prompt": ["fp8_rope_quantize_qkv", "fa_forward_raise"],
                  "prompt into a cache": ["fp8_rope_quantize_qkv_cache", "fa_forward_raise"]}[kind]
    blk = block()
    blk.eps, blk.norm1, blk.norm2 = 1e-5, torch.ones(H * HD), torch.ones(H * HD)
    blk.gate_up_interleaved = u8(1)
    blk.qkv = blk.o = blk.gate_up = blk.down = type("Layer", (), {"w": nn.FP8Tensor(u8(1), torch.ones(2))})
    blk.rope_tables = lambda S, dev: (torch.ones(S, HD // 2), torch.ones(S, HD // 2))
    blk.fa = type("Context", (), {"ptr": 1, "_msg": lambda self: "why"})()
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: type("Stream", (), {"cuda_stream": 0}))
    monkeypatch.setattr(nn, "_entry_points", lambda: (1, 2, 3, 4, 5, 6))
    monkeypatch.setattr(F, "FAStatusString", lambda status: f"status {status}")
    run = {"step": lambda: blk.decode_step(torch.zeros(B, H * HD), cache()), "prompt": lambda: blk.forward_fused(torch.zeros(B * 8, H * HD), B, 8),
           "prompt into a cache": lambda: blk.forward_fused(torch.zeros(B * 8, H * HD), B, 8, cache())}[kind]
    for place, name in enumerate(["fp8_block_run", *calls, *["fp8_gemm_rows"] * 4 * (kind == "step")]):
        def failing(*args):   # the entry points of the fields in front, that of the products of rows behind them
            assert args[:5] == (1, 2, 3, 4, 5) and args[-1] == 6 and len(args) == len(BG.BlockRunArgs._fields_) + 1
            return place << 16 | 5

        monkeypatch.setattr(BG, "BlockRun", failing)
        error = F.FAError if name.startswith("fa") else G.FP8GEMMError if name.startswith("fp8_gemm") else BG.BlockGlueError
        with pytest.raises(error) as e:
            run()
        assert type(e.value) is error and str(e.value) == (f"{name}: status 5 (why)" if error is F.FAError else f"{name}: CUDA error 5")
    blk.fa.ptr = 0
    with pytest.raises(F.FAError, match="FAContext.Decode: nil ctx" if kind == "step" else "FAContext.ForwardEx: nil ctx"):
        run()
