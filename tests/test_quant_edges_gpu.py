"""FP32 quantiser on inputs that its 32-byte loads cannot read, and on sizes around a step of a thread."""
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 8, 9, 4097, 65543, 65544, 131079, 131080, 196608, 196609, 300000, 1048575, 1048576, 1048583])
@pytest.mark.parametrize("offset", [0, 4])
def test_any_alignment_and_size(cuda, built_libs, n, offset):
    # one cluster up to 196608 values, two kernels above; one, two or four groups of 8 values in flight; offset 4: 16-byte but not 32-byte aligned
    from goml_b200 import quantize as Q
    g = torch.Generator(device="cuda").manual_seed(n)
    room = torch.randn(n + 16, generator=g, device="cuda") * 3
    x = room[offset:offset + n]
    q = torch.full((n + 32,), 0xAA, dtype=torch.uint8, device="cuda")
    words = torch.full((2,), 99.0, device="cuda")
    Q.QuantizeF32ToF8E4M3(x.data_ptr(), q.data_ptr(), words.data_ptr(), words.data_ptr() + 4, n)
    torch.cuda.synchronize()
    codes, scale, amax = O.quantize_f32(x.cpu().numpy())
    assert words.tolist() == [scale, amax]
    assert (q[:n].cpu().numpy() == codes).all() and (q[n:] == 0xAA).all()


@pytest.mark.parametrize("n", [4088, 4095, 4096, 4104, 8192, 8200, 61440, 65528])
def test_clusters_of_every_size(cuda, built_libs, n):
    # 512 groups of 8 values are one warp to a CTA of the cluster
    for offset in (0, 4):
        test_any_alignment_and_size(cuda, built_libs, n, offset)
