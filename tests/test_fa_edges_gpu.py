"""Attention forward where masks cut key blocks (every 32-key chunk of a block is masked, left alone or skipped per warp), and
where V is converted: by a pre-pass or in the kernel."""
import math
import re

import numpy as np
import pytest

import oracle as O
from tests.gpu_util import captured_nodes, has_pre_pass, kernels, run_attention

pytestmark = pytest.mark.gpu


def codes(bh, s, hd, seed):
    return [O.quantize_f32(O.seeded_normal(t, (bh, s, hd), config=f"edges{seed}"))[0] for t in "QKV"]


def near(o, lse, q, k, v, causal, window, scale):
    # P is rounded to fp16 (2^-11 of itself, so of the largest |v| at most) and O once more; the fp32 steps are far below that
    ref, lref = O.attention_f64(q, k, v, causal, window, scale)
    assert np.abs(o - ref).max() <= 2.0 ** -10 * 448 + 1e-3
    assert np.abs(o - ref).mean() <= 1e-3 * np.abs(ref).mean() + 1e-6
    assert np.abs(lse - lref).max() <= 1e-4


@pytest.mark.parametrize("scale", [1.0, -1.0])
@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("s", [1, 31, 33, 64, 97, 129, 200, 321])
def test_masks_that_cut_chunks(fa_ctx, s, hd, scale):
    q, k, v = codes(2, s, hd, s)
    scale *= 1.0 / (80.0 ** 2 * math.sqrt(hd))
    for causal in (0, 1):
        for window in sorted({w for w in (0, 1, 2, 31, 32, 33, 63, 64, 65, 96, 127, 128, 129, 160, s - 1, s) if 0 <= w <= s}):
            o, lse = run_attention(fa_ctx, q, k, v, causal, window, scale)
            near(o, lse, q, k, v, causal, window, scale)


@pytest.mark.parametrize("s,hd,causal,window", [(1025, 128, 0, 0), (1536, 128, 0, 0), (1500, 128, 1, 0), (1500, 128, 1, 1000), (1400, 64, 0, 0), (1100, 64, 1, 0),
                                                (1279, 64, 0, 700)])
def test_v_converted_ahead_and_in_the_kernel_gives_the_same_bits(cuda, built_libs, fa_ctx, s, hd, causal, window):
    # few heads have V converted by a pre-pass, more of them in the kernel; a head's result does not depend on the others
    import torch
    g = torch.Generator(device="cuda").manual_seed(s)
    q, k, v = (torch.randint(0, 0x70, (13, s, hd), generator=g, dtype=torch.uint8, device="cuda") for _ in range(3))
    for t in (q, k, v):
        t ^= torch.randint(0, 2, t.shape, generator=g, dtype=torch.uint8, device="cuda") << 7
    v[2, s - 1, 3] = 0x7f   # NaN
    out = []
    for heads in (3, 13):
        o = torch.zeros(heads, s, hd, dtype=torch.float16, device="cuda")
        lse = torch.zeros(heads, s, device="cuda")
        call = lambda: fa_ctx.ForwardEx(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr(), heads, s, hd, causal, window, 1e-5, 1.0, 0, 0, 0,
                                        torch.cuda.current_stream().cuda_stream)
        call()
        torch.cuda.synchronize()
        assert has_pre_pass(call) == (heads == 3)
        fa_ctx.DeviceStatus()
        out.append((o[:3], lse[:3]))
    assert torch.isnan(out[0][0][2, s - 1, 3]) and not torch.isnan(out[0][0][:2]).any()
    assert torch.equal(out[0][0].view(torch.int16), out[1][0].view(torch.int16)) and torch.equal(out[0][1], out[1][1])


@pytest.mark.parametrize("s,hd,causal,window", [(1, 64, 1, 0), (127, 128, 1, 0), (129, 64, 1, 0), (300, 128, 0, 0), (2700, 128, 1, 0), (2700, 64, 0, 0), (256, 128, 0, 0),
                                                (500, 64, 1, 33)])
def test_the_largest_output(cuda, built_libs, fa_ctx, s, hd, causal, window):
    # raised, not set; of the rows of the sequences alone; the output itself is the other entry point's (its kernel of masked launches
    # serves the unmasked ones here)
    import ctypes as C
    import torch
    from goml_b200 import fa_forward as F
    g = torch.Generator(device="cuda").manual_seed(s)
    q, k, v = (torch.randint(0, 0x70, (5, s, hd), generator=g, dtype=torch.uint8, device="cuda") for _ in range(3))
    v ^= torch.randint(0, 2, v.shape, generator=g, dtype=torch.uint8, device="cuda") << 7
    want, o = (torch.zeros(5, s, hd, dtype=torch.float16, device="cuda") for _ in range(2))
    fa_ctx.ForwardEx(q.data_ptr(), k.data_ptr(), v.data_ptr(), want.data_ptr(), 0, 5, s, hd, causal, window, 1e-5, 1.0)
    args = F.ForwardArgs(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), None, 5, s, hd, causal, window, 1e-5, 1.0, None, None, None, None)
    top = want.float().abs().max().item()
    for start in (0.0, 2 * top):
        word = torch.tensor([start], device="cuda")
        assert F.FALoad().fa_forward_raise(fa_ctx.ptr, C.byref(args), word.data_ptr()) == 0
        torch.cuda.synchronize()
        assert torch.equal(o, want) and word.item() == max(start, top)
    fa_ctx.DeviceStatus()
    assert F.FALoad().fa_forward_raise(fa_ctx.ptr, C.byref(args), None) == F.FA_ERR_INVALID_ARG


@pytest.mark.parametrize("s,heads,causal,window", [(129, 300, 0, 0), (1, 600, 1, 0), (255, 301, 1, 77), (64, 600, 0, 0), (2600, 30, 1, 0)])
def test_output_rows_copied_whole(cuda, built_libs, fa_ctx, s, heads, causal, window):
    # with many tiles the rows leave as copies of their own, with few as runs of a warp: the same bits, and nothing around them
    import torch
    g = torch.Generator(device="cuda").manual_seed(s)
    q, k, v = (torch.randint(0, 0x70, (heads, s, 128), generator=g, dtype=torch.uint8, device="cuda") for _ in range(3))
    room = torch.full((heads * s * 128 + 128,), 7.0, dtype=torch.float16, device="cuda")
    o = room[64:-64].view(heads, s, 128)
    run = lambda i, n, out: fa_ctx.ForwardEx(q[i:].data_ptr(), k[i:].data_ptr(), v[i:].data_ptr(), out.data_ptr(), 0, n, s, 128, causal, window, 1e-5, 1.0, 0, 0, 0,
                                             torch.cuda.current_stream().cuda_stream)
    copies = lambda n: any(re.search(r"fa_fwd_kernelILi128ELb[01]ELb[01]ELb0ELb1E", name) for name in kernels(lambda: run(0, n, o)))   # <128, .., .., false, COPY>
    assert copies(heads) and not copies(2)
    run(0, heads, o)
    for i in (0, heads - 2):
        few = torch.zeros(2, s, 128, dtype=torch.float16, device="cuda")
        run(i, 2, few)
        torch.cuda.synchronize()
        assert torch.equal(few, o[i:i + 2])
    fa_ctx.DeviceStatus()
    assert torch.isfinite(o).all() and (room[:64] == 7).all() and (room[-64:] == 7).all()


def placed(fa_ctx, heads, s, hd, causal, window=0):
    """Whether V is converted ahead, and how many CTAs of the attention's kernel an SM holds: alone, and beside a CTA of another kernel."""
    import torch
    q = torch.zeros(heads, s, hd, dtype=torch.uint8, device="cuda")
    o = torch.empty(heads, s, hd, dtype=torch.float16, device="cuda")
    p = q.data_ptr()
    nodes = captured_nodes(lambda: fa_ctx.ForwardEx(p, p, p, o.data_ptr(), 0, heads, s, hd, causal, window, 1.0, 1.0, 0, 0, 0,
                                                    torch.cuda.current_stream().cuda_stream))
    smem, = [bytes_ for _, name, bytes_ in nodes if name and "fa_fwd_kernel" in name]
    total, taken = torch.cuda.get_device_properties(0).shared_memory_per_multiprocessor, 1024   # what every CTA takes besides
    fit = lambda room: min(2, room // (smem + taken))   # registers for two
    return any(name and "v_to_f16" in name for _, name, _ in nodes), fit(total), fit(total - taken)


@pytest.mark.parametrize("heads,s,hd,causal,window", [(4, 4700, 128, 1, 0), (10, 5500, 128, 1, 0), (8, 4790, 64, 1, 0), (24, 4096, 128, 0, 0), (70, 8192, 64, 0, 0)])
def test_tiles_in_front_are_spread_while_the_pre_pass_runs(cuda, built_libs, fa_ctx, heads, s, hd, causal, window):
    ahead, alone, beside = placed(fa_ctx, heads, s, hd, causal, window)
    assert ahead and beside == 1 and alone in (1, 2)


@pytest.mark.parametrize("heads,s,hd,causal,window,alone", [(5, 4000, 64, 1, 0, 1), (8, 3000, 64, 1, 3000, 1), (4, 4700, 128, 1, 0, 1), (1, 1, 64, 1, 0, 1),
                                                            (16, 1664, 64, 1, 0, 1), (16, 1792, 64, 1, 0, 2), (17, 1000, 128, 1, 0, 2), (8, 2500, 64, 1, 500, 2),
                                                            (8, 2500, 128, 0, 0, 2)])
def test_few_long_tiles_have_an_sm_each(cuda, built_libs, fa_ctx, heads, s, hd, causal, window, alone):
    # 148 SMs: up to 222 tiles of up to 16 heads; and the same bits either way, one head at a time among them
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert sms == 148
    assert placed(fa_ctx, heads, s, hd, causal, window)[1] == alone
    g = torch.Generator(device="cuda").manual_seed(s)
    q, k, v = (torch.randint(0, 0x70, (heads, s, hd), generator=g, dtype=torch.uint8, device="cuda") for _ in range(3))
    o, one = torch.empty(heads, s, hd, dtype=torch.float16, device="cuda"), torch.empty(s, hd, dtype=torch.float16, device="cuda")
    run = lambda n, i, out: fa_ctx.ForwardEx(q[i:].data_ptr(), k[i:].data_ptr(), v[i:].data_ptr(), out.data_ptr(), 0, n, s, hd, causal, window, 1e-5, 1.0)
    run(heads, 0, o)
    for i in (0, heads - 1):
        run(1, i, one)
        torch.cuda.synchronize()
        assert torch.equal(one, o[i])
    fa_ctx.DeviceStatus()


@pytest.mark.parametrize("heads", [15, 16, 17, 29, 30, 32, 33, 47, 300])
@pytest.mark.parametrize("s,hd,window", [(129, 128, 0), (400, 64, 0), (400, 128, 100), (1800, 64, 0)])
def test_tiles_of_heads_in_one_group_or_several(cuda, built_libs, fa_ctx, heads, s, hd, window):
    # every tile of every head once: a head's bits do not depend on the heads beside it
    import torch
    if heads * s > 100_000:
        heads = 100_000 // s
    g = torch.Generator(device="cuda").manual_seed(heads)
    q, k, v = (torch.randint(0, 0x70, (heads, s, hd), generator=g, dtype=torch.uint8, device="cuda") for _ in range(3))
    o, few = (torch.full((heads, s, hd), 7.0, dtype=torch.float16, device="cuda") for _ in range(2))
    run = lambda i, n, out: fa_ctx.ForwardEx(q[i:].data_ptr(), k[i:].data_ptr(), v[i:].data_ptr(), out[i:].data_ptr(), 0, n, s, hd, 1, window, 1e-5, 1.0)
    run(0, heads, o)
    for i in range(0, heads, 5):
        run(i, min(5, heads - i), few)
    torch.cuda.synchronize()
    fa_ctx.DeviceStatus()
    assert torch.equal(o, few)


@pytest.mark.parametrize("s,hd,causal,window", [(64, 64, 0, 0), (64, 128, 0, 0), (192, 128, 0, 0), (256, 64, 0, 0), (320, 64, 0, 0), (1600, 128, 0, 0), (2752, 64, 0, 0),
                                                (1, 64, 1, 0), (130, 128, 1, 0), (1000, 128, 1, 200), (2700, 128, 1, 0), (4300, 64, 1, 0)])
def test_a_walk_over_tiles_gives_what_single_tiles_give(cuda, built_libs, fa_ctx, s, hd, causal, window):
    # more tiles than CTAs fit: tiles of one block, of an odd number and of many, behind one another in a CTA; both signs of the scale.  A few
    # heads at a time have a CTA per tile: the same bits, LSE and largest output
    import ctypes as C
    import torch
    from goml_b200 import fa_forward as F
    tiles = (s + 127) // 128
    heads = 900 // tiles + 1
    g = torch.Generator(device="cuda").manual_seed(s + hd)
    q, k, v = (torch.randint(0, 0x70, (heads, s, hd), generator=g, dtype=torch.uint8, device="cuda") for _ in range(3))
    q ^= torch.randint(0, 2, q.shape, generator=g, dtype=torch.uint8, device="cuda") << 7
    o, few, raised = (torch.full((heads, s, hd), 7.0, dtype=torch.float16, device="cuda") for _ in range(3))
    lse, few_lse = (torch.full((heads, s), 7.0, device="cuda") for _ in range(2))
    run = lambda i, n, out, l, scale: fa_ctx.ForwardEx(q[i:].data_ptr(), k[i:].data_ptr(), v[i:].data_ptr(), out[i:].data_ptr(), l[i:].data_ptr(), n, s, hd, causal,
                                                       window, scale, 1.0, 0, 0, 0, torch.cuda.current_stream().cuda_stream)
    walking = lambda n: any(re.search(r"fa_fwd_kernelILi\d+ELb[01]ELb[01]ELb0ELb1E", name) for name in kernels(lambda: run(0, n, o, lse, 1.0)))   # <.., false, WALK>
    step = max(1, 200 // tiles)
    assert walking(heads) and not walking(step)
    for scale in (1e-4, -1e-4):
        run(0, heads, o, lse, scale)
        for i in range(0, heads, step):
            run(i, min(step, heads - i), few, few_lse, scale)
        args = F.ForwardArgs(q.data_ptr(), k.data_ptr(), v.data_ptr(), raised.data_ptr(), None, heads, s, hd, causal, window, scale, 1.0, None, None, None, None)
        word = torch.zeros(1, device="cuda")
        assert F.FALoad().fa_forward_raise(fa_ctx.ptr, C.byref(args), word.data_ptr()) == 0
        torch.cuda.synchronize()
        fa_ctx.DeviceStatus()
        assert torch.equal(o, few) and torch.equal(lse, few_lse) and torch.equal(o, raised) and word.item() == o.float().abs().max().item()
