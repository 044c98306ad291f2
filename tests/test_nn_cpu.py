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
