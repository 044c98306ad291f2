"""Kernels that start before their predecessor on the stream has drained: chains of dependent calls, queued without a
synchronisation and over the same buffers, give what the same calls give one at a time."""
import math

import pytest
import torch

from tests.gpu_util import has_pre_pass, kernels

pytestmark = pytest.mark.gpu
STEPS = 50


def twice(step, out):
    """step(i) -> None writes out[i]: once with a synchronisation behind every step, once queued behind a short pause so that
    the whole chain runs back to back on the GPU."""
    got = []
    for queued in (False, True):
        out.fill_(0)
        torch.cuda.synchronize()
        if queued:
            torch.cuda._sleep(30_000_000)   # some 15 ms
        for i in range(STEPS):
            step(i)
            if not queued:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        got.append(out.clone())
    assert torch.equal(*got)
    return got[0]


@pytest.mark.parametrize("B,S,H,hd,ahead", [(1, 40, 2, 64, False), (2, 300, 8, 128, False), (1, 700, 6, 64, False), (1, 1300, 4, 128, True), (1, 1100, 2, 64, True),
                                            (1, 2700, 9, 128, True)])
def test_rope_quantise_then_attention(cuda, built_libs, fa_ctx, B, S, H, hd, ahead):
    # V and the scales of every step are written by the kernel right ahead of the attention, one cluster or two kernels; with V
    # converted in the attention's kernel, and by a pre-pass that hands it on chunk by chunk
    from goml_b200 import block_glue as BG
    g = torch.Generator(device="cuda").manual_seed(S)
    qkv = [(torch.randn(B * S, 3, H, hd, generator=g, device="cuda") * (0.1 + i % 7)).bfloat16() for i in range(STEPS)]
    cos, sin = (torch.empty(S, hd // 2, device="cuda") for _ in range(2))
    BG.RopeTable(cos.data_ptr(), sin.data_ptr(), S, hd, 10000.0)
    q, k, v = (torch.empty(B * H, S, hd, dtype=torch.uint8, device="cuda") for _ in range(3))
    s6 = torch.empty(6, device="cuda")
    out = torch.empty(STEPS, B * H, S, hd, dtype=torch.float16, device="cuda")
    sp, stream = s6.data_ptr(), torch.cuda.current_stream().cuda_stream

    def step(i):
        BG.RopeQuantizeQKV(qkv[i].data_ptr(), cos.data_ptr(), sin.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), sp, sp + 12, B, S, H, hd, stream)
        fa_ctx.ForwardEx(q.data_ptr(), k.data_ptr(), v.data_ptr(), out[i].data_ptr(), 0, B * H, S, hd, 1, 0, 1.0 / math.sqrt(hd), 1.0,
                         sp, sp + 4, sp + 8, stream)

    got = twice(step, out)
    assert has_pre_pass(lambda: fa_ctx.ForwardEx(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), 0, B * H, S, hd, 1, 0, 1.0, 1.0, 0, 0, 0,
                                                 torch.cuda.current_stream().cuda_stream)) == ahead
    # the first query of a sequence sees one key: its output is that key's V, 2^-4 relative to a code and its fp16 rounding
    want = torch.stack([x.view(B, S, 3, H, hd)[:, 0, 2].reshape(B * H, hd).float() for x in qkv])
    assert ((got[:, :, 0].float() - want).abs() <= 0.07 * want.abs() + 2e-3 * want.abs().amax(dim=(1, 2), keepdim=True)).all()


@pytest.mark.parametrize("B,Hq,Hkv,hd,paged", [(2, 4, 4, 64, False), (3, 8, 2, 128, True), (30, 32, 32, 128, False), (24, 32, 8, 128, True)])
def test_append_then_decode(cuda, built_libs, fa_ctx, B, Hq, Hkv, hd, paged):
    # the q scale, the appended rows and the lengths of every step are written by the kernel right ahead of the decode attention
    from goml_b200 import block_glue as BG
    g = torch.Generator(device="cuda").manual_seed(B)
    s_max, page = 256, 64
    qkv = [(torch.randn(B, (Hq + 2 * Hkv) * hd, generator=g, device="cuda") * (0.1 + i % 7)).bfloat16() for i in range(STEPS)]
    cos, sin = (torch.empty(s_max, hd // 2, device="cuda") for _ in range(2))
    BG.RopeTable(cos.data_ptr(), sin.data_ptr(), s_max, hd, 10000.0)
    per = s_max // page
    table = torch.randperm(B * per, generator=g, device="cuda").to(torch.int32).view(B, per)
    shape = (B * per, Hkv, page, hd) if paged else (B, Hkv, s_max, hd)
    k, v = (torch.empty(shape, dtype=torch.uint8, device="cuda") for _ in range(2))
    k0, v0 = (torch.randint(0, 0x60, shape, generator=g, dtype=torch.uint8, device="cuda") for _ in range(2))
    lens0 = (torch.arange(B, device="cuda") * 17 % 150).to(torch.int32)
    lens = torch.empty_like(lens0)
    q = torch.empty(B, Hq, hd, dtype=torch.uint8, device="cuda")
    qs, kvs = torch.empty(2, device="cuda"), torch.tensor([0.02, 0.03], device="cuda")
    out = torch.empty(STEPS, B, Hq, hd, dtype=torch.float16, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    more = dict(block_table=table.data_ptr(), page_size=page, max_pages_per_seq=per, num_pages=B * per) if paged else {}

    def step(i):
        if i == 0:
            k.copy_(k0), v.copy_(v0), lens.copy_(lens0)
        BG.DecodeRopeAppend(qkv[i].data_ptr(), cos.data_ptr(), sin.data_ptr(), lens.data_ptr(), q.data_ptr(), qs.data_ptr(), qs.data_ptr() + 4,
                            k.data_ptr(), v.data_ptr(), kvs.data_ptr(), kvs.data_ptr() + 4, B, Hq, Hkv, hd, 0 if paged else s_max, s_max,
                            seq_lens_out=lens.data_ptr(), stream=stream, **more)
        fa_ctx.Decode(q.data_ptr(), k.data_ptr(), v.data_ptr(), out[i].data_ptr(), 0, lens.data_ptr(), B, Hq, Hkv, hd, 0 if paged else s_max, 0,
                      1.0 / math.sqrt(hd), 1.0, qs.data_ptr(), kvs.data_ptr(), kvs.data_ptr() + 4, stream, **more)

    twice(step, out)
    assert torch.isfinite(out).all() and lens.tolist() == [n + STEPS for n in lens0.tolist()]


@pytest.mark.parametrize("B,H,hd,paged", [(1, 32, 128, False), (4, 32, 128, True), (9, 32, 128, False), (9, 32, 64, True), (1, 16, 64, False)])
def test_append_then_decode_in_clusters(cuda, built_libs, fa_ctx, B, H, hd, paged):
    # splits of 256 rows that meet in clusters of two to four: sequences of 1 to 186 keys, which the first of them has all, or some of them
    x = torch.zeros(B * H * 256 * hd, dtype=torch.uint8, device="cuda")
    lens = torch.full((B,), 7, dtype=torch.int32, device="cuda")
    name, = kernels(lambda: fa_ctx.Decode(x.data_ptr(), x.data_ptr(), x.data_ptr(), torch.empty(B, H, hd, dtype=torch.float16, device="cuda").data_ptr(), 0, lens.data_ptr(),
                                          B, H, H, hd, 256, 0, 1.0, 1.0, stream=torch.cuda.current_stream().cuda_stream))
    assert "fa_decode_kernel" in name and name.split("EvN")[0].endswith("Lb1EE")
    test_append_then_decode(cuda, built_libs, fa_ctx, B, H, H, hd, paged)


@pytest.mark.parametrize("M,K,F,N,variant", [(300, 512, 704, 520, "Li64ELi1"), (1000, 1024, 1376, 517, "Li256ELi1"), (2048, 2048, 4736, 520, "Li256ELi2")])
def test_quantise_then_square_gemm(cuda, built_libs, M, K, F, N, variant):
    # norm + quantiser -> gate/up GEMM -> quantiser -> GEMM into 16 bits, rows of whole pieces and odd ones -> and the next step's norm
    # into the codes that the first GEMM has just read; every kernel overlaps the one ahead
    from goml_b200 import block_glue as BG, fp8_gemm as G
    g = torch.Generator(device="cuda").manual_seed(M)
    xs = [torch.randn(M, K, generator=g, device="cuda") * (0.1 + i) for i in range(5)]
    code = lambda rows, k: torch.randn(rows, k, generator=g, device="cuda").mul_(2).to(torch.float8_e4m3fn).view(torch.uint8)
    w1, w2 = G.interleave_gate_up(code(2 * F, K), F), code(N, F)
    gamma = [1 + torch.randn(K, generator=g, device="cuda") * 0.3 for _ in range(STEPS)]
    empty = lambda *shape, dtype=torch.uint8: torch.empty(shape, dtype=dtype, device="cuda")
    codes, hb, hc, rstd, w = empty(M, K), empty(M, F, dtype=torch.bfloat16), empty(M, F), empty(M, dtype=torch.float32), empty(5, dtype=torch.float32)
    out = empty(STEPS, M, N, dtype=torch.bfloat16)
    p, stream = w.data_ptr(), torch.cuda.current_stream().cuda_stream
    weight_scale = torch.full((1,), 2.0 ** -7, device="cuda")
    up = lambda: G.FP8GEMMSwiGLURaise(M, F, K, codes.data_ptr(), w1.data_ptr(), hb.data_ptr(), 1.0, p, weight_scale.data_ptr(), p + 8,
                                      torch.cuda.current_stream().cuda_stream)

    def step(i):
        BG.RMSNormQuantizeInto(xs[i % 5].data_ptr(), 0, gamma[i].data_ptr(), codes.data_ptr(), p, p + 4, rstd.data_ptr(), p + 8, M, K, 1e-5, stream)
        up()
        BG.QuantizeBF16(hb.data_ptr(), hc.data_ptr(), p + 12, p + 8, M * F, stream)
        G.FP8GEMMScaled(M, N, F, hc.data_ptr(), w2.data_ptr(), out[i].data_ptr(), 1.0, p + 12, weight_scale.data_ptr(), G.OutBF16, stream)

    got = twice(step, out)
    assert G.device_status() == 0
    name, = kernels(up)
    assert f"fp8_gemm_tcgen05_kernelI{variant}E" in name
    # the last step against its own codes: bf16 rounding of the result, and of the sums' last bits
    want = hc.view(torch.float8_e4m3fn).double() @ w2.view(torch.float8_e4m3fn).double().t() * w[3].double() * 2.0 ** -7
    assert ((got[-1].double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5 * want.abs().max()).all()


@pytest.mark.parametrize("B,d,H,Fh", [(1, 512, 4, 1376), (2, 512, 8, 1376), (1, 2048, 16, 5504)])
def test_steps_behind_rewritten_weights(cuda, built_libs, B, d, H, Fh):
    # the products of a step of one or two sequences load their weights ahead of the wait, all but the first one's: every step's weights
    # and scales are written by the kernels right ahead of it, those of its last product last
    from goml_b200 import fp8_gemm as G, nn
    g = torch.Generator(device="cuda").manual_seed(d + B)
    rn = lambda *shape: torch.randn(*shape, generator=g, device="cuda") * 0.02
    blk = nn.FP8DecoderBlock(d, H, Fh, rn(3 * d, d), rn(d, d), rn(2 * Fh, d), rn(d, Fh), 1 + rn(d), 1 + rn(d))
    held = lambda b: [b.qkv.w.codes, b.o.w.codes, b.gate_up_interleaved, b.qkv.w.sa, b.o.w.sa, b.gate_up.w.sa, b.down.w.sa, b.down.w.codes]
    sets = []
    for i in range(3):
        other = nn.FP8DecoderBlock(d, H, Fh, *(rn(*shape) * (0.5 + i) for shape in ((3 * d, d), (d, d), (2 * Fh, d), (d, Fh))), 1 + rn(d), 1 + rn(d))
        sets.append([w.clone() for w in held(other)])
        other.close()
    xs = torch.randn(STEPS, B, d, generator=g, device="cuda")
    cache = nn.FP8KVCache(B, H, STEPS + 8, d // H)
    cache.scales.fill_(0.02)
    out = torch.empty(STEPS, B, d, device="cuda")

    def step(i):
        if i == 0:
            for buf in (cache.k, cache.v, cache.lens):
                buf.zero_()
        for w, new in zip(held(blk), sets[i % 3]):
            w.copy_(new)
        out[i].copy_(blk.decode_step(xs[i], cache))

    got = twice(step, out)
    assert got.isfinite().all() and cache.lens.tolist() == [STEPS] * B and G.device_status() == 0
    assert sum("fp8_gemm_skinny_kernel" in n and "ELb1E" in n for n in kernels(lambda: blk.decode_step(xs[0], cache))) == 4
    blk.close()
