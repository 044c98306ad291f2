"""FP8 GEMM where the output's rows are not whole 16-byte pieces, and on both sides of the few-row kernel's lines: products of
-1, 0 and 1, whose sums are whole numbers that fp16 holds, so every element is compared exactly."""
import re

import pytest
import torch

from tests.gpu_util import kernels

pytestmark = pytest.mark.gpu


def exact(M, N, K, offset=0, out="fp16", seed=0):
    from goml_b200 import fp8_gemm as G
    g = torch.Generator(device="cuda").manual_seed(seed + 1000 * M + N)
    a, b = (torch.randint(-1, 2, (rows, K), generator=g, device="cuda") for rows in (M, N))
    codes = lambda x: torch.tensor([0xb8, 0x00, 0x38], dtype=torch.uint8, device="cuda")[x + 1].contiguous()
    ad, bd = codes(a), codes(b)
    dtype = torch.float16 if out == "fp16" else torch.bfloat16
    room = torch.full((M * N + 64,), 7.0, dtype=dtype, device="cuda")
    c = room[16 + offset:16 + offset + M * N]
    G.FP8GEMMScaled(M, N, K, ad.data_ptr(), bd.data_ptr(), c.data_ptr(), 1.0, 0, 0, G.OutFP16 if out == "fp16" else G.OutBF16, 0)
    torch.cuda.synchronize()
    assert G.device_status() == 0
    want = a.double() @ b.double().t()
    assert torch.equal(c.view(M, N).double(), want.to(dtype).double())
    assert (room[:16 + offset] == 7).all() and (room[16 + offset + M * N:] == 7).all()   # nothing around it


@pytest.mark.parametrize("N", [1, 2, 3, 5, 31, 62, 63, 64, 65, 66, 67, 127, 130, 191, 252, 255, 257, 260, 513, 1001])
@pytest.mark.parametrize("M", [193, 257])
def test_rows_of_any_length(cuda, built_libs, M, N):
    for offset in (0, 1, 2, 4):   # elements past a 16-byte boundary
        exact(M, N, 64, offset)
    exact(M, N, 64, 0, "bf16")


@pytest.mark.parametrize("M,N,K", [(4097, 517, 128), (700, 5555, 256), (300, 20003, 2048), (5000, 2001, 2048)])
def test_many_tiles_with_rows_of_any_length(cuda, built_libs, M, N, K):
    # tiles of every width, halves of a short last wave and tile pairs
    exact(M, N, K)


@pytest.mark.parametrize("M", [81, 100, 128, 129, 150, 192])
@pytest.mark.parametrize("N,K", [(1024, 2992), (1024, 3008), (1501, 4784), (1501, 4800), (130, 8192)])
def test_few_rows_on_both_sides_of_the_lines(cuda, built_libs, M, N, K):
    exact(M, N, K)


@pytest.mark.parametrize("M,N,K,offset,few", [(100, 1024, 8192, 0, False), (150, 2048, 5504, 0, False), (192, 512, 8192, 0, False), (81, 2048, 3008, 0, False),
                                              (80, 1024, 8192, 0, True), (100, 1023, 8192, 0, True), (100, 1024, 8192, 1, True), (128, 4096, 11008, 0, True),
                                              (150, 3008, 8000, 0, True), (193, 512, 8192, 0, False)])
def test_added_to_fp32_by_the_kernel_that_cuts_a_long_k_best(cuda, built_libs, M, N, K, offset, few):
    # offset: values past a 16-byte boundary, where the copy engine cannot add and the square kernel does not cut K
    from goml_b200 import fp8_gemm as G
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a, b = (torch.randint(-1, 2, (rows, K), generator=g, device="cuda") for rows in (M, N))
    codes = lambda x: torch.tensor([0xb8, 0x00, 0x38], dtype=torch.uint8, device="cuda")[x + 1].contiguous()
    ad, bd = codes(a), codes(b)
    room = torch.full((M * N + 64,), 7.0, device="cuda")
    x = room[16 + offset:16 + offset + M * N].view(M, N)
    x.copy_(torch.randint(-9, 10, (M, N), generator=g, device="cuda").float())
    want = x.double() + a.double() @ b.double().t()
    call = lambda: G.FP8GEMMAccumulateF32(M, N, K, ad.data_ptr(), bd.data_ptr(), x.data_ptr(), 1.0, 0, 0, torch.cuda.current_stream().cuda_stream)
    name, = kernels(call)
    assert ("skinny" in name) == few
    call()
    torch.cuda.synchronize()
    assert G.device_status() == 0 and torch.equal(x.double(), want)
    assert (room[:16 + offset] == 7).all() and (room[16 + offset + M * N:] == 7).all()


@pytest.mark.parametrize("M,N,K,variant", [(512, 5000, 2048, "Li192ELi1"), (390, 5000, 2064, "Li192ELi1"), (1024, 5000, 6000, "Li192ELi2"), (900, 5184, 6000, "Li192ELi2"),
                                           (700, 8192, 4096, "Li192ELi2"), (1500, 5000, 4096, "Li256ELi2")])
def test_units_that_fill_their_waves(cuda, built_libs, M, N, K, variant):
    # tiles and pairs of 192 columns: last pairs half empty, last columns of less than a tile; 16-bit results of both types, added to fp32, and the bits
    # that single tiles of 256 columns give
    from goml_b200 import fp8_gemm as G
    stream = lambda: torch.cuda.current_stream().cuda_stream
    exact(M, N, K)
    exact(M, N, K, 0, "bf16")
    g = torch.Generator(device="cuda").manual_seed(M)
    a, b = (torch.randint(0, 0x78, (rows, K), generator=g, dtype=torch.uint8, device="cuda") for rows in (M, N))
    s = torch.tensor([3e-3, 2e-3], device="cuda")
    x0 = torch.randn(M, N, generator=g, device="cuda")

    def outputs():
        c, x = torch.empty(M, N, dtype=torch.bfloat16, device="cuda"), x0.clone()
        calls = [lambda: G.FP8GEMMScaled(M, N, K, a.data_ptr(), b.data_ptr(), c.data_ptr(), 1.0, s.data_ptr(), s.data_ptr() + 4, G.OutBF16, stream()),
                 lambda: G.FP8GEMMAccumulateF32(M, N, K, a.data_ptr(), b.data_ptr(), x.data_ptr(), 1.0, s.data_ptr(), s.data_ptr() + 4, stream())]
        names = [n for call in calls for n in kernels(call)]
        for call in calls:
            call()
        torch.cuda.synchronize()
        assert G.device_status() == 0
        return names, c, x

    names, c, x = outputs()
    assert len(names) == 2 and all(f"tcgen05_kernelI{variant}E" in n for n in names)
    G.SetTilePairs(0)
    try:
        others, c1, x1 = outputs()
    finally:
        G.SetTilePairs(-1)
    assert all("ELi1E" in n for n in others)
    assert torch.equal(c, c1) and torch.equal(x, x1)
    # rows that leave through no tensor map keep the shape that they had
    name, = kernels(lambda: G.FP8GEMMScaled(M, N - 1, K, a.data_ptr(), b.data_ptr(), c.data_ptr(), 1.0, 0, 0, G.OutBF16, stream()))
    assert "Li192" not in name


def unit_of(call):
    """(columns, tiles) of the work units that a product's kernel has."""
    name, = kernels(call)
    return tuple(int(n) for n in re.search(r"tcgen05_kernelILi(\d+)ELi(\d)E", name).groups())


@pytest.mark.parametrize("M,N,K,swiglu,offset,unit", [(1500, 4992, 4096, False, 0, (256, 2)), (1500, 4992, 4096, False, 1, (256, 1)), (1500, 4992, 4096, False, 8, (256, 1)),
                                                      (2431, 960, 2256, False, 0, (256, 1)), (1725, 5184, 6096, True, 0, (256, 2)), (1725, 5184, 6096, True, 1, (256, 1)),
                                                      (1725, 5181, 6096, True, 0, (256, 1))])
def test_results_that_no_map_describes_keep_their_units(cuda, built_libs, M, N, K, swiglu, offset, unit):
    # e4m3 results and activations, offset by values past a 16-byte boundary: pairs pay the longer end in full, and tiles of 64 columns have no map
    from goml_b200 import fp8_gemm as G
    g = torch.Generator(device="cuda").manual_seed(M + offset)
    rows = 2 * ((N + 31) // 32) * 32 if swiglu else N
    a, b = (torch.randint(0, 0x78, (n, K), generator=g, dtype=torch.uint8, device="cuda") for n in (M, rows))
    s = torch.tensor([3e-3, 2e-3, 1e-2], device="cuda")
    p, stream = s.data_ptr(), lambda: torch.cuda.current_stream().cuda_stream

    def result(offset):
        room = torch.full((M * N + 64,), 3, dtype=torch.bfloat16 if swiglu else torch.uint8, device="cuda")
        out, top = room[16 + offset:16 + offset + M * N], torch.zeros(1, device="cuda")
        if swiglu:
            call = lambda: G.FP8GEMMSwiGLURaise(M, N, K, a.data_ptr(), b.data_ptr(), out.data_ptr(), 1.0, p, p + 4, top.data_ptr(), stream())
        else:
            call = lambda: G.FP8GEMMFP8Out(M, N, K, a.data_ptr(), b.data_ptr(), out.data_ptr(), 1.0, p, p + 4, p + 8, top.data_ptr(), stream())
        took = unit_of(call)
        call()
        torch.cuda.synchronize()
        assert G.device_status() == 0
        assert (room[:16 + offset] == 3).all() and (room[16 + offset + M * N:] == 3).all()
        return took, out.view(torch.uint8), top

    took, out, top = result(offset)
    assert took == unit
    G.SetTilePairs(0)
    try:
        single, want, want_top = result(0)
    finally:
        G.SetTilePairs(-1)
    assert single[1] == 1 and torch.equal(out, want) and torch.equal(top, want_top)


# what a unit of another shape promises is not kept: a short K; pairs for single tiles or tiles of 128 columns, single tiles for pairs, as rows begin; narrow tiles
@pytest.mark.parametrize("kind,M,N,K,unit", [("c", 1213, 2560, 240, (256, 1)), ("c", 1213, 2560, 256, (192, 1)), ("x", 1213, 2560, 112, (256, 1)), ("x", 1213, 2560, 128, (192, 1)),
                                             ("c", 4096, 4096, 128, (256, 1)), ("c", 4096, 4096, 4096, (256, 1)), ("d", 4096, 4096, 4096, (256, 1)), ("c", 4096, 4096, 3072, (256, 1)),
                                             ("c", 4096, 4096, 3088, (256, 2)), ("c", 4192, 2080, 5888, (128, 1)), ("c", 4192, 2080, 5904, (192, 2)), ("c", 1411, 6192, 1984, (128, 1)),
                                             ("c", 3524, 19360, 2160, (256, 2)), ("c", 3524, 19360, 2176, (256, 1)), ("d", 10176, 160, 4208, (256, 1))])
def test_units_that_lose_are_not_taken(cuda, built_libs, kind, M, N, K, unit):
    from goml_b200 import fp8_gemm as G
    a, b = (torch.full((rows, K), 0x38, dtype=torch.uint8, device="cuda") for rows in (M, N))
    out = torch.zeros(M, N, dtype={"c": torch.bfloat16, "x": torch.float32, "d": torch.uint8}[kind], device="cuda")
    ptrs, stream = (a.data_ptr(), b.data_ptr(), out.data_ptr()), lambda: torch.cuda.current_stream().cuda_stream
    call = {"c": lambda: G.FP8GEMMScaled(M, N, K, *ptrs, 1.0, 0, 0, G.OutBF16, stream()), "x": lambda: G.FP8GEMMAccumulateF32(M, N, K, *ptrs, 1.0, 0, 0, stream()),
            "d": lambda: G.FP8GEMMFP8Out(M, N, K, *ptrs, 1.0 / K, 0, 0, 0, 0, stream())}[kind]
    assert unit_of(call) == unit
    call()
    torch.cuda.synchronize()
    assert G.device_status() == 0
    want = torch.tensor(K, dtype=torch.float32).to(out.dtype) if kind != "d" else 0x38   # ones: sums of K, or 1 as a code
    assert (out == want).all()


@pytest.mark.parametrize("split,K", [(1, 384), (2, 512), (3, 880), (4, 1024), (5, 6400), (6, 7696), (7, 8960), (8, 10240)])
@pytest.mark.parametrize("N", [200, 131])
def test_sums_handed_to_their_owners_and_fetched_are_the_same(cuda, built_libs, split, K, N):
    # up to 16 rows a CTA's sums go to their owner, past that the owners fetch them: added in the same order, so every row has the same bits
    from goml_b200 import fp8_gemm as G
    g = torch.Generator(device="cuda").manual_seed(split + N)
    a, b = (torch.randint(0, 0x70, (rows, K), generator=g, dtype=torch.uint8, device="cuda") for rows in (17, 2 * ((N + 31) // 32) * 32))
    a ^= torch.randint(0, 2, a.shape, generator=g, dtype=torch.uint8, device="cuda") << 7
    s = torch.tensor([3e-3, 2e-3], device="cuda")
    sa, sb = s.data_ptr(), s.data_ptr() + 4
    x0 = torch.randn(17, N, generator=g, device="cuda")

    def outputs(M):
        st = torch.cuda.current_stream().cuda_stream
        c, x, h = torch.empty(M, N, dtype=torch.bfloat16, device="cuda"), x0[:M].clone(), torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
        d, top = torch.empty(M, N, dtype=torch.uint8, device="cuda"), torch.zeros(2, device="cuda")
        calls = [lambda: G.FP8GEMMScaled(M, N, K, a.data_ptr(), b.data_ptr(), c.data_ptr(), 1.0, sa, sb, G.OutBF16, torch.cuda.current_stream().cuda_stream),
                 lambda: G.FP8GEMMAccumulateF32(M, N, K, a.data_ptr(), b.data_ptr(), x.data_ptr(), 1.0, sa, sb, st),
                 lambda: G.FP8GEMMSwiGLURaise(M, N, K, a.data_ptr(), b.data_ptr(), h.data_ptr(), 1.0, sa, sb, top.data_ptr(), st),
                 lambda: G.FP8GEMMFP8Out(M, N, K, a.data_ptr(), b.data_ptr(), d.data_ptr(), 1.0, sa, sb, 0, top.data_ptr() + 4, st)]
        name, = kernels(calls[0])
        assert f"ILi{split}ELb0ELi{int(M <= 16)}E" in name
        for call in calls:
            call()
        torch.cuda.synchronize()
        assert G.device_status() == 0 and top[0].item() == h.float().abs().max().item() and top[1].item() > 0
        return c, x, h, d

    whole = outputs(17)
    for M in (1, 2, 15, 16):
        for got, want in zip(outputs(M), whole):
            assert torch.equal(got.view(torch.uint8), want[:M].contiguous().view(torch.uint8))
    ref = lambda t: t.view(torch.float8_e4m3fn).double()
    want = 6e-6 * ref(a) @ ref(b[:N]).t()
    # a product of 17 bits a term, summed in fp32: 2^-24 a sum, and bf16's 2^-9
    assert ((whole[0].double() - want).norm() / want.norm()).item() < 4e-3


@pytest.mark.parametrize("M,K,few", [(80, 3008, True), (100, 3008, False), (128, 3488, False), (128, 3504, True), (150, 4784, False), (150, 4800, True)])
def test_codes_on_both_sides_of_the_line(cuda, built_libs, M, K, few):
    from goml_b200 import fp8_gemm as G
    N = 1024
    g = torch.Generator(device="cuda").manual_seed(M)
    a, b = (torch.randint(-1, 2, (rows, K), generator=g, device="cuda") for rows in (M, N))
    codes = lambda x: torch.tensor([0xb8, 0x00, 0x38], dtype=torch.uint8, device="cuda")[x + 1].contiguous()
    ad, bd = codes(a), codes(b)
    d, amax = torch.empty(M, N, dtype=torch.uint8, device="cuda"), torch.zeros(1, device="cuda")
    call = lambda: G.FP8GEMMFP8Out(M, N, K, ad.data_ptr(), bd.data_ptr(), d.data_ptr(), 1.0, 0, 0, 0, amax.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert ("skinny" in "".join(kernels(call))) == few
    call()
    torch.cuda.synchronize()
    want = (a.double() @ b.double().t())
    assert amax.item() == want.abs().max().item()
    assert torch.equal(d.view(torch.float8_e4m3fn).float(), want.float().to(torch.float8_e4m3fn).float())


@pytest.mark.parametrize("shape", [(1, 64), (3, 5, 64), (64,), (200, 64)])
def test_linear_layer_takes_any_tensor(cuda, built_libs, shape):
    # contiguous fp32 goes straight to the libraries, everything else through views and copies: the same bits
    import torch
    from goml_b200 import nn
    g = torch.Generator(device="cuda").manual_seed(len(shape))
    layer = nn.FP8Linear(torch.randn(40, 64, generator=g, device="cuda"))
    x = torch.randn(shape, generator=g, device="cuda").bfloat16().float()
    want = layer.forward_codes(nn.quantize(x.reshape(-1, 64)), x.numel() // 64)
    strided = torch.stack([x, x + 1], -1)[..., 0]
    assert not strided.is_contiguous() and want.shape == (x.numel() // 64, 40)
    for same in (x, strided, x.bfloat16(), x.double(), x.clone().requires_grad_()):
        assert torch.equal(layer(same), want)
    with pytest.raises(RuntimeError):
        layer(torch.zeros(65, device="cuda"))
    with pytest.raises(AssertionError):
        layer(x.cpu())
    with pytest.raises(Exception):
        layer(torch.zeros(0, 64, device="cuda"))
