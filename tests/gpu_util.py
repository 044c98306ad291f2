"""Helpers for the GPU parity tests: torch is used for device memory only."""
import ctypes as C

import numpy as np
import torch


def dev_u8(a: np.ndarray) -> torch.Tensor:
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.uint8)).cuda()


def run_gemm(a, b, alpha=None, bf16=True, scale_ptrs=(0, 0), entry="scaled"):
    """C = A.B^T through the C ABI on e4m3 code arrays; returns a numpy float64 array."""
    from goml_b200 import fp8_gemm as G
    M, K = a.shape
    N = b.shape[0]
    ad, bd = dev_u8(a), dev_u8(b)
    c = torch.full((M, N), float("nan"), dtype=torch.bfloat16 if bf16 else torch.float16, device="cuda")
    if entry == "scaled":
        G.FP8GEMMScaled(M, N, K, ad.data_ptr(), bd.data_ptr(), c.data_ptr(), 1.0 if alpha is None else alpha,
                        scale_ptrs[0], scale_ptrs[1], G.OutBF16 if bf16 else G.OutFP16, 0)
    elif entry == "gemm":
        G.FP8GEMM(M, N, K, ad.data_ptr(), bd.data_ptr(), c.data_ptr(), 1, 0)
    elif entry == "original":
        G.FP8GEMMOriginal(M, N, K, ad.data_ptr(), bd.data_ptr(), c.data_ptr(), 0)
    else:
        G.FP8GEMMSinglesync(M, N, K, ad.data_ptr(), bd.data_ptr(), c.data_ptr(), 0)
    torch.cuda.synchronize()
    assert G.device_status() == 0
    return c.double().cpu().numpy()


def run_attention(ctx, q, k, v, causal=0, window=0, scale=None, v_descale=1.0, entry="train", want_lse=True):
    """Attention through the C ABI on e4m3 code arrays [bh, sl, hd]; returns (O f64, LSE f64 or None)."""
    import math
    bh, sl, hd = q.shape
    if scale is None:
        scale = 1.0 / math.sqrt(hd)
    qd, kd, vd = dev_u8(q), dev_u8(k), dev_u8(v)
    o = torch.zeros((bh, sl, hd), dtype=torch.float16, device="cuda")          # zero-initialised as the
    lse = torch.zeros((bh, sl), dtype=torch.float32, device="cuda") if want_lse else None  # reference callers do
    lp = lse.data_ptr() if want_lse else 0
    if entry == "train":
        ctx.ForwardTrain(qd.data_ptr(), kd.data_ptr(), vd.data_ptr(), o.data_ptr(), lp, bh, sl, hd, causal, window, scale, 0)
    elif entry == "forward":
        ctx.Forward(qd.data_ptr(), kd.data_ptr(), vd.data_ptr(), o.data_ptr(), bh, sl, hd, causal, window, scale, 0)
    else:
        ctx.ForwardEx(qd.data_ptr(), kd.data_ptr(), vd.data_ptr(), o.data_ptr(), lp, bh, sl, hd, causal, window, scale, v_descale)
    torch.cuda.synchronize()
    ctx.DeviceStatus()
    return o.double().cpu().numpy(), (lse.double().cpu().numpy() if want_lse and entry != "forward" else None)


class _KernelParams(C.Structure):   # CUDA_KERNEL_NODE_PARAMS_v2
    _fields_ = [("func", C.c_void_p)] + [(n, C.c_uint) for n in ("gx", "gy", "gz", "bx", "by", "bz", "smem")] + \
               [(n, C.c_void_p) for n in ("params", "extra", "kern", "ctx")]


def captured_nodes(call):
    """The nodes that call() leaves in a graph: (CUgraphNodeType, name of the kernel or None, its dynamic shared memory) each."""
    cu = C.CDLL("libcuda.so.1")
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=torch.cuda.Stream()):
        call()
    n = C.c_size_t()
    raw = C.c_void_p(graph.raw_cuda_graph())
    assert cu.cuGraphGetNodes(raw, None, C.byref(n)) == 0
    nodes = (C.c_void_p * n.value)()
    assert cu.cuGraphGetNodes(raw, nodes, C.byref(n)) == 0
    out = []
    for node in nodes:
        t, name, p = C.c_int(), None, _KernelParams()
        assert cu.cuGraphNodeGetType(C.c_void_p(node), C.byref(t)) == 0
        if t.value == 0:
            text = C.c_char_p()
            assert cu.cuGraphKernelNodeGetParams_v2(C.c_void_p(node), C.byref(p)) == 0
            got = cu.cuFuncGetName(C.byref(text), C.c_void_p(p.func)) if p.func else cu.cuKernelGetName(C.byref(text), C.c_void_p(p.kern))
            assert got == 0
            name = text.value.decode()
        out.append((t.value, name, p.smem))
    return out


def kernels(call):
    """Names (as the linker knows them) of the kernels that call() launches."""
    return [name for _, name, _ in captured_nodes(call) if name]


def has_pre_pass(call):
    """Whether an attention call has V converted ahead of its kernel."""
    names = kernels(call)
    assert sum("fa_fwd_kernel" in n for n in names) == 1
    return any("v_to_f16_kernel" in n for n in names)
