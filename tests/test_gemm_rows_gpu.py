"""Products that quantise their few rows themselves (fp8_gemm_rows), against a quantiser and the product behind it."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu
NOT_SUPPORTED, INVALID = 801, 1


def call(lib, **fields):
    from goml_b200 import fp8_gemm as G
    import torch
    return lib.fp8_gemm_rows(C.byref(G.RowsArgs(stream=torch.cuda.current_stream().cuda_stream, **fields)))


# the blocks' products, with n as the width of the SwiGLU too; few and many tiles, slices of one to four, two and three CTAs to an SM; K ragged in 128 and 64; N ragged in 128 and 4
@pytest.mark.parametrize("m,n,k", [(1, 12288, 4096), (2, 4096, 4096), (2, 22016, 4096), (2, 4096, 11008), (1, 2048, 5504), (2, 1001, 2000), (1, 128, 16), (1, 6144, 2048),
                                   (2, 8192, 8192), (2, 11264, 2048), (1, 130, 272), (1, 11008, 4096),
                                   (2, 11008, 4096), (2, 5504, 2048), (1, 5632, 2048)])
@pytest.mark.parametrize("source", [1, 2, 3])
def test_rows_against_quantiser_and_product(cuda, built_libs, m, n, k, source):
    import torch
    from goml_b200 import block_glue as BG, fp8_gemm as G, quantize as Q
    lib = G._init()
    g = torch.Generator(device="cuda").manual_seed(n + k + m)
    x = torch.randn(m, k, generator=g, device="cuda") * 3
    x[:, k // 2] *= 7     # a row maximum that is not everywhere
    gamma = 1 + 0.1 * torch.randn(k, generator=g, device="cuda")
    w = torch.randint(0, 0x70, (2 * ((n + 31) // 32) * 32, k), generator=g, dtype=torch.uint8, device="cuda")
    w ^= torch.randint(0, 2, w.shape, generator=g, dtype=torch.uint8, device="cuda") << 7
    ws = torch.tensor([1e-3], device="cuda")
    codes, words = torch.empty(m, k, dtype=torch.uint8, device="cuda"), torch.zeros(64, device="cuda")
    p, st = words.data_ptr(), torch.cuda.current_stream().cuda_stream
    if source == 1:
        rows = x
        BG.RMSNormQuantizeInto(x.data_ptr(), 0, gamma.data_ptr(), codes.data_ptr(), p, p + 4, torch.empty(m, device="cuda").data_ptr(), 0, m, k, 1e-5, st)
    else:
        rows = x.to(torch.float16 if source == 2 else torch.bfloat16)
        f = rows.float()
        Q.QuantizeF32ToF8E4M3(f.data_ptr(), codes.data_ptr(), p, p + 4, f.numel(), st)
    more = dict(rows=rows.data_ptr(), gamma=gamma.data_ptr() if source == 1 else None, amax=p + 4 if source == 3 else None, scale_b=ws.data_ptr(), m=m, k=k, source=source,
                eps=1e-5, b=w.data_ptr())
    # an RMSNorm adds its squares in another order: the scale may differ in the last bits, and a code by a step here and there
    rel = 2e-3 if source == 1 else 1e-6

    def close(got, want, out_eps):
        d = (got.double() - want.double()).norm() / want.double().norm()
        assert d <= rel + out_eps, d.item()

    # bf16 outputs, and words that are cleared
    want, c = torch.empty(m, n, dtype=torch.bfloat16, device="cuda"), torch.full((m + 1, n), 7.0, dtype=torch.bfloat16, device="cuda")
    G.FP8GEMMScaled(m, n, k, codes.data_ptr(), w.data_ptr(), want.data_ptr(), 1.0, p, ws.data_ptr(), G.OutBF16, st)
    zero = torch.full((40,), 3.0, device="cuda")
    assert call(lib, c=c.data_ptr(), n=n, zero=zero.data_ptr(), zeros=33, **more) == 0
    close(c[:m], want, 1e-3 if source == 1 else 2e-4)   # another order of the sums: neighbouring bf16 values, rarely
    assert (c[m] == 7).all() and (zero[:33] == 0).all() and (zero[33:] == 3).all()
    # added to another matrix, and to one in place
    base = torch.randn(m, n, generator=g, device="cuda")
    want32, out, inplace = base.clone(), torch.full((m + 1, n), 7.0, device="cuda"), base.clone()
    G.FP8GEMMAccumulateF32(m, n, k, codes.data_ptr(), w.data_ptr(), want32.data_ptr(), 1.0, p, ws.data_ptr(), st)
    assert call(lib, x=out.data_ptr(), x_in=base.data_ptr(), n=n, b_complete=0, **more) == 0
    torch.cuda.synchronize()
    assert call(lib, x=inplace.data_ptr(), x_in=inplace.data_ptr(), n=n, b_complete=1, **more) == 0
    close(out[:m], want32, 1e-6)
    assert torch.equal(out[:m], inplace) and (out[m] == 7).all()
    # SwiGLU, its maximum raised
    wh, h, top = torch.empty(m, n, dtype=torch.bfloat16, device="cuda"), torch.empty(m, n, dtype=torch.bfloat16, device="cuda"), torch.zeros(2, device="cuda")
    G.FP8GEMMSwiGLU(m, n, k, codes.data_ptr(), w.data_ptr(), wh.data_ptr(), 1.0, p, ws.data_ptr(), top.data_ptr(), st)
    rc = call(lib, h=h.data_ptr(), h_amax=top.data_ptr() + 4, n=n, b_complete=1, **more)
    assert rc == (NOT_SUPPORTED if (n, k) == (22016, 4096) else 0)   # 344 tiles of weight rows: more than two to an SM
    if rc == 0:
        close(h, wh, 4e-3 if source == 1 else 1e-3)
        assert top[1].item() == h.float().abs().max().item()
    torch.cuda.synchronize()
    assert G.device_status() == 0


# as many k-blocks to a CTA as leave two stages: 192 of a whole K, of two and three slices, 77 where two CTAs share an SM, 39 of two slices where three do; one more is refused
@pytest.mark.parametrize("m,n,k,taken", [(2, 14336, 24576, True), (1, 14336, 24576, True), (2, 14336, 24592, False), (2, 7680, 49152, True), (1, 5120, 73728, True), (2, 5120, 73728, True),
                                         (2, 30720, 9856, True), (2, 30720, 9872, False), (2, 20480, 9984, True), (2, 20480, 10000, False)])
def test_the_longest_rows(cuda, built_libs, m, n, k, taken):
    # 448 times -1, 0 or 1 has the scale 1, and the sums with weights of -1, 0 and 1 are multiples of 448 that fp32 holds
    import torch
    from goml_b200 import fp8_gemm as G
    lib = G._init()
    g = torch.Generator(device="cuda").manual_seed(n + k + m)
    ones = lambda *shape: torch.randint(-1, 2, shape, generator=g, dtype=torch.int8, device="cuda")
    x, w = ones(m, k), ones(n, k)
    x[:, 0] = 1
    rows = (448 * x.float()).half()
    codes = torch.where(w == 0, 0, torch.where(w > 0, 0x38, 0xb8)).to(torch.uint8)
    base, one = torch.randint(-50, 50, (m, n), generator=g, device="cuda").float(), torch.ones(1, device="cuda")
    out = torch.full((m + 1, n), 7.0, device="cuda")
    rc = call(lib, rows=rows.data_ptr(), b=codes.data_ptr(), scale_b=one.data_ptr(), x=out.data_ptr(), x_in=base.data_ptr(), m=m, n=n, k=k, source=G.RowsF16)
    torch.cuda.synchronize()
    assert G.device_status() == 0
    assert rc == (0 if taken else NOT_SUPPORTED)
    want = base.double() + 448 * torch.stack([torch.cat([(x[j:j + 1] * part).sum(1, dtype=torch.int32) for part in w.split(1024)]) for j in range(m)])
    assert torch.equal(out[:m].double(), want if taken else torch.full_like(want, 7.0)) and (out[m] == 7).all()


# n a multiple of four or not, whole and cut tiles; sizes that need four slices and one
@pytest.mark.parametrize("m,n,k", [(1, 4096, 4096), (2, 1000, 2048), (2, 1001, 2000)])
def test_the_stream_may_lie_on_any_four_bytes(cuda, built_libs, m, n, k):
    # x_in and x each 0 to 12 bytes past a multiple of 16: the same bits, nothing written around x
    import torch
    from goml_b200 import fp8_gemm as G
    lib = G._init()
    g = torch.Generator(device="cuda").manual_seed(n)
    rows = torch.randn(m, k, generator=g, device="cuda").half()
    w = torch.randint(0, 0x70, (n, k), generator=g, dtype=torch.uint8, device="cuda")
    ws = torch.tensor([1e-3], device="cuda")
    base = torch.randn(m, n, generator=g, device="cuda")
    src, dst = (torch.empty(m * n + 8, device="cuda") for _ in range(2))
    assert src.data_ptr() % 16 == dst.data_ptr() % 16 == 0
    got = []
    for i in range(4):
        for j in range(4):
            src.fill_(9.0)
            src[i:i + m * n].copy_(base.view(-1))
            dst.fill_(7.0)
            assert call(lib, rows=rows.data_ptr(), b=w.data_ptr(), scale_b=ws.data_ptr(), x=dst.data_ptr() + 4 * j, x_in=src.data_ptr() + 4 * i, m=m, n=n, k=k,
                        source=G.RowsF16) == 0
            got.append(dst[j:j + m * n].clone())
            assert (dst[:j] == 7).all() and (dst[j + m * n:] == 7).all()
    torch.cuda.synchronize()
    assert G.device_status() == 0
    assert not torch.equal(got[0], base.view(-1)) and all(torch.equal(got[0], other) for other in got)


def test_values_without_a_scale_and_beyond_numbers(cuda, built_libs):
    # all zeros: scale 1.  NaN never wins the maximum and gets the code that the quantiser's clamp makes of it, -448
    import torch
    from goml_b200 import fp8_gemm as G
    lib = G._init()
    n, k = 1024, 2048
    w = torch.full((n, k), 0x38, dtype=torch.uint8, device="cuda")   # ones
    one = torch.ones(1, device="cuda")
    x = torch.zeros(2, k, dtype=torch.float16, device="cuda")
    c = torch.empty(2, n, dtype=torch.bfloat16, device="cuda")
    args = dict(b=w.data_ptr(), scale_b=one.data_ptr(), rows=x.data_ptr(), c=c.data_ptr(), m=2, n=n, k=k, source=G.RowsF16)
    assert call(lib, **args) == 0
    assert (c == 0).all()
    x[0, :8], x[1, 5] = 1.0, float("nan")
    assert call(lib, **args) == 0
    assert (c[0] == 8).all() and (c[1] == -1).all()
    torch.cuda.synchronize()
    assert G.device_status() == 0


def test_what_is_refused(cuda, built_libs):
    import torch
    from goml_b200 import fp8_gemm as G
    lib = G._init()
    buf = torch.zeros(1 << 22, dtype=torch.uint8, device="cuda")
    p = buf.data_ptr()
    good = dict(rows=p, gamma=p, b=p + (1 << 16), scale_b=p + 64, c=p + (1 << 21), m=1, n=256, k=1024, source=1, eps=1e-5)
    assert call(lib, **good) == 0
    assert lib.fp8_gemm_rows(None) == INVALID
    for bad in (dict(rows=None), dict(b=None), dict(gamma=None), dict(source=0), dict(source=4), dict(k=1000), dict(k=0), dict(m=-1), dict(n=-1), dict(c=None), dict(x=p, x_in=p),
                dict(c=None, x=p + (1 << 21)), dict(c=None, h=p + (1 << 21)), dict(source=3), dict(zeros=1), dict(zeros=65, zero=p), dict(rows=p + 8), dict(b=p + 8),
                dict(gamma=p + 4), dict(c=p + 1)):
        assert call(lib, **{**good, **bad}) == INVALID, bad
    assert call(lib, **{**good, "m": 3}) == NOT_SUPPORTED
    torch.cuda.synchronize()
    assert G.device_status() == 0
