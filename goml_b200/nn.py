"""FP8 dispatch of goml's nn call sites for one Llama-style decoder block (prefill).

goml's `nn.Linear.Forward` (nn/linear.go:53-74), `nn.FeedForward.forwardSwiGLU`
(nn/feedforward.go:54-79: W2(silu(W1 x) * W3 x)) and `nn.MultiHeadAttention.Forward`
(nn/attention.go:60-160) run in F32 today.  Here every projection goes through the FP8
GEMM library, the attention through the FP8 attention library and every quantisation
through the quantiser library — scales stay on the device between them (no host round
trip).  The row-local glue (RMSNorm with eps inside the square root, half-split RoPE, SiLU
gate, residual adds, layout permutes: the arithmetic of
internal/abjexam/llama_hf_f64ref.go:126-178 and battle_a_llm_f64ref.go:182-237) runs
through libfp8block.so, each op fused with the quantiser of the next GEMM / attention
operand (`fused=True`, the default), or as plain fp32 torch ops followed by separate
quantiser calls (`fused=False`, kept as the unfused comparison).

torch tensors are used as device buffers; all heavy kernels are reached through the C ABI.
"""
from __future__ import annotations

import ctypes
import math

import torch

from . import block_glue as BG, fa_forward as F, fp8_gemm as G, quantize as Q


class FP8Tensor:
    """e4m3 codes + a one-float device scale (and the amax word the quantiser writes)."""

    def __init__(self, codes: torch.Tensor, scale_amax: torch.Tensor):
        self.codes = codes
        self.sa = scale_amax  # [scale, amax] fp32 on the device

    @property
    def scale_ptr(self) -> int:
        return self.sa.data_ptr()


def quantize(x: torch.Tensor, unit: bool = False) -> FP8Tensor:
    """Per-tensor FP32 -> e4m3 through libfp8quant (scale = amax/448, or amax when unit)."""
    x = x.contiguous()
    assert x.dtype == torch.float32 and x.is_cuda
    codes = torch.empty(x.shape, dtype=torch.uint8, device=x.device)
    sa = torch.empty(2, dtype=torch.float32, device=x.device)   # both written by the quantiser
    fn = Q.QuantizeF32ToF8E4M3Unit if unit else Q.QuantizeF32ToF8E4M3
    fn(x.data_ptr(), codes.data_ptr(), sa.data_ptr(), sa.data_ptr() + 4, x.numel(), torch.cuda.current_stream().cuda_stream)
    return FP8Tensor(codes, sa)


class FP8Linear:
    """y = x W^T with W [out, in] (the layout of nn/linear.go:14), both operands e4m3, bf16 result."""

    def __init__(self, weight: torch.Tensor):
        self.out_features, self.in_features = weight.shape
        self.w = quantize(weight.float())

    def __call__(self, x: torch.Tensor) -> torch.Tensor:
        M, K = x.numel() // self.in_features, self.in_features
        if (x.dtype is not torch.float32 or not x.is_cuda or x.numel() != M * K or not x.is_contiguous()
                or type(self).forward_codes is not FP8Linear.forward_codes or "forward_codes" in vars(self)):   # a layer with a product of its own has it called
            return self.forward_codes(quantize(x.reshape(M, K).float()), M)
        # codes, scale and amax in one allocation and no views: for a few rows a call is its host time (28.7 us with a tensor for each)
        buf, codes, sa = _scratch(x.device, M * K, 8)
        stream = torch.cuda.current_stream().cuda_stream
        Q.QuantizeF32ToF8E4M3(x.data_ptr(), codes, sa, sa + 4, M * K, stream)
        return self._product(codes, sa, M, x.device, stream)

    def accumulate_into(self, xq: FP8Tensor, M: int, x: torch.Tensor) -> None:
        """x (fp32 [M, out]) += this layer's output, added in the GEMM epilogue (no 16-bit intermediate)."""
        assert x.dtype == torch.float32 and x.is_contiguous() and x.shape == (M, self.out_features)
        G.FP8GEMMAccumulateF32(M, self.out_features, self.in_features, xq.codes.data_ptr(), self.w.codes.data_ptr(), x.data_ptr(),
                               1.0, xq.scale_ptr, self.w.scale_ptr, torch.cuda.current_stream().cuda_stream)

    def forward_codes(self, xq: FP8Tensor, M: int) -> torch.Tensor:
        """The GEMM alone, on an activation that is already e4m3 codes + device scale."""
        return self._product(xq.codes.data_ptr(), xq.scale_ptr, M, xq.codes.device, torch.cuda.current_stream().cuda_stream)

    def _product(self, codes: int, scale: int, M: int, device: torch.device, stream: int) -> torch.Tensor:
        y = torch.empty((M, self.out_features), dtype=torch.bfloat16, device=device)
        G.FP8GEMMScaled(M, self.out_features, self.in_features, codes, self.w.codes.data_ptr(), y.data_ptr(),
                        1.0, scale, self.w.scale_ptr, G.OutBF16, stream)
        return y


def rms_norm(x: torch.Tensor, gamma: torch.Tensor, eps: float) -> torch.Tensor:
    return gamma * x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps)


def rope_half_split(x: torch.Tensor, theta: float) -> torch.Tensor:
    """x [B, H, S, hd]: pairs (i, i + hd/2), angle = pos * theta^(-2i/hd)."""
    hd, S = x.shape[-1], x.shape[-2]
    half = hd // 2
    freq = theta ** (-2.0 * torch.arange(half, device=x.device, dtype=torch.float64) / hd)
    ang = torch.arange(S, device=x.device, dtype=torch.float64)[:, None] * freq[None, :]
    c, s = ang.cos().float(), ang.sin().float()
    x0, x1 = x[..., :half], x[..., half:]
    return torch.cat([x0 * c - x1 * s, x0 * s + x1 * c], dim=-1)


class FP8KVCache:
    """One layer's FP8 KV cache: K and V codes [batch, heads, s_max, hd] with one dequantisation scale each, fixed
    when the prompt is written, and the per-sequence lengths on the device.  The structure of the KVCache sketched in
    goml's runs/reports/F1_HF_INFERENCE_recon.md:186-196 (Append at position tCur, K()/V() views), holding e4m3 codes
    instead of fp32 and S_max allocated up front."""

    def __init__(self, batch: int, heads: int, s_max: int, hd: int, device="cuda"):
        self.B, self.H, self.s_max, self.hd = batch, heads, s_max, hd
        self.k = torch.zeros((batch, heads, s_max, hd), dtype=torch.uint8, device=device)
        self.v = torch.zeros_like(self.k)
        self.scales = torch.ones(2, dtype=torch.float32, device=device)      # k_scale, v_scale
        self.lens = torch.zeros(batch, dtype=torch.int32, device=device)     # keys cached per sequence

    def dense_on(self, device: torch.device) -> bool:
        """Whether kernels of `device` that are given the buffers' pointers find the cache there: codes [batch, heads, s_max, hd]
        without gaps, two scales and the lengths, all on that device."""
        k, v, scales, lens = self.k, self.v, self.scales, self.lens
        if not (k.device == v.device == scales.device == lens.device == device and scales.dtype is torch.float32 and lens.dtype is torch.int32
                and k.is_contiguous() and v.is_contiguous() and scales.is_contiguous() and lens.is_contiguous()):
            return False
        if k.shape == v.shape == (self.B, self.H, self.s_max, self.hd) and k.dtype is v.dtype is torch.uint8 and lens.shape == (self.B,):
            return scales.numel() >= 2
        # other views of the same bytes
        codes = self.B * self.H * self.s_max * self.hd
        return (all(t.element_size() == 1 and t.numel() >= codes and (t.dim() == 1 or t.shape[-2:] == (self.s_max, self.hd)) for t in (k, v))
                and scales.numel() >= 2 and lens.numel() >= self.B)

    def takes(self, batch: int, heads: int, S: int, hd: int, device: "torch.device | None" = None) -> bool:
        """Whether a prompt's codes can be written straight into this cache by a kernel of `device` (the codes' own by default)."""
        device = self.k.device if device is None else device
        k, v = self.k, self.v
        return (batch == self.B and heads == self.H and hd == self.hd and S <= self.s_max and self.dense_on(device)
                and k.shape == v.shape == (batch, heads, self.s_max, hd) and k.dtype is v.dtype is torch.uint8
                and (k.data_ptr() | v.data_ptr()) % 16 == 0 and self.scales.shape == (2,) and self.lens.shape == (batch,))

    def fill(self, k_codes, v_codes, scales, S: int) -> None:
        """Prompt phase: K/V codes [batch*heads, S, hd] as the prefill quantiser wrote them, and their two scales."""
        self.k[:, :, :S].copy_(k_codes.view(self.B, self.H, S, self.hd))
        self.v[:, :, :S].copy_(v_codes.view(self.B, self.H, S, self.hd))
        self.scales.copy_(scales)
        self.lens.fill_(S)


def _writes_directly(cache, B: int, H: int, S: int, hd: int, device: torch.device) -> bool:
    """Whether the prompt's codes go straight into the cache; a cache with a `fill` of its own has that called."""
    return isinstance(cache, FP8KVCache) and type(cache).fill is FP8KVCache.fill and "fill" not in vars(cache) and cache.takes(B, H, S, hd, device)


def _scratch(dev, *sizes):
    """One allocation cut into 256-byte aligned pieces: (the buffer, their addresses).  A call has a dozen temporaries, and
    drawing each from the allocator took about a third of a decode step's host time."""
    offsets, total = [], 0
    for n in sizes:
        offsets.append(total)
        total += (n + 255) & -256
    buf = torch.empty(total, dtype=torch.uint8, device=dev)
    base = buf.data_ptr()
    return (buf, *[base + o for o in offsets])


_entries = None


def _entry_points():
    """Addresses of the library entry points that fp8_block_run calls."""
    global _entries
    if _entries is None:
        gemm, fa = G._init(), F.FALoad()
        _entries = tuple(ctypes.cast(fn, ctypes.c_void_p).value for fn in (gemm.fp8_gemm_scaled, gemm.fp8_gemm_accumulate_f32, gemm.fp8_gemm_swiglu_raise,
                                                                           fa.fa_forward_raise, fa.fa_decode, gemm.fp8_gemm_rows))
    return _entries


def _stream_start(x: torch.Tensor, rows: int, d: int):
    """(source, h) of a block's residual stream: h is written by the first RMSNorm while it reads x, or is a copy already
    (source = h) where x is not what that kernel reads.  The kernels behind it address h as rows of d values without gaps, so
    what its copy does not turn into that (a clone keeps the order of strides) is refused."""
    assert x.shape == (rows, d), f"the block takes [{rows}, {d}], not {list(x.shape)}"
    if (x.dtype == torch.float32 and x.is_contiguous() and x.data_ptr() % 32 == 0
            and not (x.requires_grad and torch.is_grad_enabled())):
        return x, torch.empty_like(x)
    h = x.float().clone()
    assert h.is_contiguous(), f"the block takes rows of {d} values, not strides {x.stride()}"
    return h, h


class FP8DecoderBlock:
    """Llama-style block: RMSNorm -> QKV -> RoPE -> causal FP8 attention -> O -> residual -> RMSNorm -> SwiGLU -> residual."""

    def __init__(self, d_model, n_heads, ffn_hidden, wqkv, wo, wgate_up, wdown, norm1, norm2, eps=1e-5, theta=10000.0, fused=True):
        self.fused = fused
        self._rope = {}   # seq_len -> (cos, sin) device tables
        self.d, self.H, self.F = d_model, n_heads, ffn_hidden
        self.hd = d_model // n_heads
        assert self.hd in (64, 128)
        self.qkv, self.o = FP8Linear(wqkv), FP8Linear(wo)
        self.gate_up, self.down = FP8Linear(wgate_up), FP8Linear(wdown)
        # the same gate/up codes in the layout the SwiGLU GEMM epilogue reads (gate and up rows of a column block adjacent)
        self.gate_up_interleaved = G.interleave_gate_up(self.gate_up.w.codes, ffn_hidden)
        self.norm1, self.norm2 = norm1.float(), norm2.float()
        self.eps, self.theta = eps, theta
        self.fa = F.FACreate()

    def attention(self, xn: torch.Tensor, B: int, S: int) -> torch.Tensor:
        H, hd = self.H, self.hd
        qkv = self.qkv(xn).float().view(B, S, 3, H, hd).permute(2, 0, 3, 1, 4)  # [3, B, H, S, hd]
        q = rope_half_split(qkv[0], self.theta)
        k = rope_half_split(qkv[1], self.theta)
        qq, kq, vq = quantize(q), quantize(k), quantize(qkv[2])
        o = torch.empty((B * H, S, hd), dtype=torch.float16, device=xn.device)
        self.fa.ForwardEx(qq.codes.data_ptr(), kq.codes.data_ptr(), vq.codes.data_ptr(), o.data_ptr(), 0, B * H, S, hd, 1, 0,
                          1.0 / math.sqrt(hd), 1.0, qq.scale_ptr, kq.scale_ptr, vq.scale_ptr, torch.cuda.current_stream().cuda_stream)
        return o.view(B, H, S, hd).permute(0, 2, 1, 3).reshape(B * S, H * hd)

    def rope_tables(self, S: int, dev) -> tuple[torch.Tensor, torch.Tensor]:
        if S not in self._rope:
            cos = torch.empty((S, self.hd // 2), dtype=torch.float32, device=dev)
            sin = torch.empty_like(cos)
            BG.RopeTable(cos.data_ptr(), sin.data_ptr(), S, self.hd, self.theta, torch.cuda.current_stream().cuda_stream)
            self._rope[S] = (cos, sin)
        return self._rope[S]

    def _run(self, x: torch.Tensor, B: int, S: int, tables: int, cache: "FP8KVCache | None", decode: bool):
        """The block's library calls (fp8_block_run): the new stream, and the scratch with the addresses of the prompt's K and V
        codes and of their scales."""
        T, d, H, Fh = B * S, self.d, self.H, self.F
        n = T * d
        up = lambda size: (size + 255) & -256
        # what the attention half needs (projections, Q codes, attention output, its codes) and then the feed-forward half
        # (activations, their codes) in the same place
        region_bytes = max(up(6 * n) + 2 * up(n) + up(2 * n), up(2 * T * Fh) + up(T * Fh))
        kv = 0 if decode else n
        buf, words, rstd, codes, kc, vc, region = _scratch(x.device, 256, 4 * T, n, kv, kv, region_bytes)
        src, h = _stream_start(x, T, d)                         # residual stream, updated in place
        cos, sin = self.rope_tables(tables, x.device)
        if not self.fa.ptr:
            raise F.FAError(f"FAContext.{'Decode' if decode else 'ForwardEx'}: nil ctx", F.FA_ERR_INVALID_ARG)
        k = v = ks = lens = s_max = 0
        if cache is not None:
            k, v, ks, lens, s_max = cache.k.data_ptr(), cache.v.data_ptr(), cache.scales.data_ptr(), cache.lens.data_ptr(), cache.s_max
        qkv, o, gate_up, down = self.qkv.w, self.o.w, self.gate_up.w, self.down.w
        *entries, gemm_rows = _entry_points()
        rc = BG.BlockRun(*entries, self.fa.ptr, src.data_ptr(), h.data_ptr(), self.norm1.data_ptr(),
                         self.norm2.data_ptr(), qkv.codes.data_ptr(), o.codes.data_ptr(), self.gate_up_interleaved.data_ptr(), down.codes.data_ptr(),
                         qkv.scale_ptr, o.scale_ptr, gate_up.scale_ptr, down.scale_ptr, cos.data_ptr(), sin.data_ptr(), k, v, ks, lens,
                         words, rstd, codes, kc, vc, region, region_bytes, torch.cuda.current_stream().cuda_stream,
                         B, S, d, H, Fh, s_max, tables, int(decode), self.eps, 1.0 / math.sqrt(self.hd), gemm_rows)
        if rc:
            self._raise(rc, decode, cache is not None)
        return h, buf, kc, vc, words + 72

    def _raise(self, rc: int, decode: bool, cached: bool) -> None:
        """The error of the library call that fp8_block_run stopped at, as its own binding raises it."""
        place, code = rc >> 16, rc & 0xffff
        if place == 4:
            raise F.FAError("fa_decode" if decode else "fa_forward_raise", code, self.fa._msg())
        if place > 10:
            raise G.FP8GEMMError(f"fp8_gemm_rows: CUDA error {code}")
        rope = "fp8_decode_rope_append" if decode else "fp8_rope_quantize_qkv_cache" if cached else "fp8_rope_quantize_qkv"
        name = ("fp8_block_run", "fp8_rmsnorm_quantize_into", "fp8_gemm_scaled", rope, "", "fp8_permute_quantize_heads",
                "fp8_gemm_accumulate_f32", "fp8_rmsnorm_quantize_into", "fp8_gemm_swiglu_raise", "fp8_quantize_bf16", "fp8_gemm_accumulate_f32")[place]
        if name.startswith("fp8_gemm"):
            raise G.FP8GEMMError(f"{name}: CUDA error {code}")
        raise BG.BlockGlueError(f"{name}: CUDA error {code}")

    def forward_fused(self, x: torch.Tensor, B: int, S: int, cache: "FP8KVCache | None" = None) -> torch.Tensor:
        """The block with every glue op fused with the quantiser of its consumer and both residual adds done in
        the GEMM epilogues, SwiGLU in the gate/up GEMM's epilogue: 10 library calls, issued in native code, no torch math.
        With `cache`, the K and V codes of the prompt and their scales are also stored there for decode_step."""
        direct = _writes_directly(cache, B, self.H, S, self.hd, x.device)
        h, buf, kc, vc, kv_scales = self._run(x, B, S, S, cache if direct else None, False)
        if cache is not None and not direct:
            view = lambda p, nbytes: buf[p - buf.data_ptr():p - buf.data_ptr() + nbytes]
            n = B * S * self.d
            cache.fill(view(kc, n), view(vc, n), view(kv_scales, 8).view(torch.float32), S)
        return h

    def decode_step(self, x: torch.Tensor, cache: FP8KVCache) -> torch.Tensor:
        """One new token per sequence: x [batch, d] fp32 -> [batch, d] fp32, the token's K and V appended to `cache` at
        position cache.lens[b] (quantised with the cache's scales) and cache.lens advanced.  Ten library calls:
        RMSNorm+quantise -> QKV GEMM -> RoPE+quantise+append -> decode attention -> quantise -> O GEMM (residual in the
        epilogue) -> the feed-forward half of forward_fused; six for one or two sequences, whose GEMMs quantise their rows themselves."""
        B = x.shape[0]
        assert (B, self.H, self.hd) == (cache.B, cache.H, cache.hd)
        if not cache.dense_on(x.device):
            raise ValueError(f"decode_step: the cache's buffers must lie without gaps, in the shapes it was made with, on {x.device}")
        # the lengths advance in place, on the device: the step can be replayed from a CUDA graph
        return self._run(x, B, 1, cache.s_max, cache, True)[0]

    def __call__(self, x: torch.Tensor, B: int, S: int, cache: "FP8KVCache | None" = None) -> torch.Tensor:
        """x [B*S, d] fp32 -> [B*S, d] fp32."""
        assert cache is None or self.fused, "the KV cache is written by the fused path"
        if self.fused:
            return self.forward_fused(x, B, S, cache)
        x = x.float()
        x = x + self.o(self.attention(rms_norm(x, self.norm1, self.eps), B, S)).float()
        gu = self.gate_up(rms_norm(x, self.norm2, self.eps)).float()
        g, u = gu[:, : self.F], gu[:, self.F:]
        x = x + self.down(torch.nn.functional.silu(g) * u).float()
        return x

    def close(self):
        self.fa.Destroy()


def _main():
    """Times the full-size block config: d_model 4096, 32 heads x 128, SwiGLU hidden 11008, B=8 x S=2048
    tokens, random-init weights N(0, 0.02), embeddings N(0, 1) — the whole block and its FP8 kernels alone."""
    import os
    import sys
    B, S, d, H, Fh = 8, 2048, 4096, 32, 11008
    if len(sys.argv) > 1:
        B = int(sys.argv[1])
    # Under torchrun the block is sharded by rows on sequence boundaries (the M-tile partition of the GEMMs and the
    # batch*head partition of the attention coincide there): weights replicated, no collective on the data path;
    # torch.distributed is used for the barrier and the max-over-ranks of the timing only.
    world, rank = int(os.environ.get("WORLD_SIZE", "1")), int(os.environ.get("RANK", "0"))
    if world > 1:
        import torch.distributed as dist
        from .multi_gpu import shard_rows
        local = int(os.environ.get("LOCAL_RANK", "0"))
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", device_id=torch.device("cuda", local))
        lo, hi = shard_rows(B * S, world, rank, tile=S)      # whole sequences per rank
        B_global, B = B, (hi - lo) // S
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(4)
    rn = lambda *shape, std=0.02: torch.randn(*shape, generator=g, device=dev) * std
    blk = FP8DecoderBlock(d, H, Fh, rn(3 * d, d), rn(d, d), rn(2 * Fh, d), rn(d, Fh), torch.ones(d, device=dev), torch.ones(d, device=dev))
    x = rn(B * S, d, std=1.0)

    def timed(fn, iters=5):
        for _ in range(2):
            fn()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(iters):
            fn()
        e1.record()
        torch.cuda.synchronize()
        return e0.elapsed_time(e1) / iters

    if world > 1:
        dist.barrier()
        t = torch.tensor([timed(lambda: blk(x, B, S), iters=10)], device=dev)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        if rank == 0:
            fl = 2.0 * B_global * S * d * (3 * d + d + 3 * Fh) + 2.0 * B_global * H * S * S * (d // H)
            print(f"block B={B_global} S={S} d={d} H={H} F={Fh} over {world} GPUs ({B} sequences per GPU, no collective): "
                  f"{t.item():.3f} ms (max over ranks) = {fl / t.item() / 1e9:.0f} TFLOPS whole job")
        blk.close()
        dist.destroy_process_group()
        return
    total = timed(lambda: blk(x, B, S))
    blk.fused = False
    total_unfused = timed(lambda: blk(x, B, S))
    blk.fused = True
    M = B * S
    # kernels alone, on pre-quantised operands
    xq = quantize(x)
    sh = torch.cuda.current_stream().cuda_stream

    def gemm(lin, a):
        y = torch.empty((M, lin.out_features), dtype=torch.bfloat16, device=dev)
        return timed(lambda: G.FP8GEMMScaled(M, lin.out_features, lin.in_features, a.codes.data_ptr(), lin.w.codes.data_ptr(),
                                             y.data_ptr(), 1.0, a.scale_ptr, lin.w.scale_ptr, G.OutBF16, sh))

    hq = quantize(rn(M, Fh, std=1.0))
    t_qkv, t_o, t_gu, t_dn = gemm(blk.qkv, xq), gemm(blk.o, xq), gemm(blk.gate_up, xq), gemm(blk.down, hq)
    hd = d // H
    q3 = [quantize(rn(B * H, S, hd, std=1.0)) for _ in range(3)]
    o = torch.empty((B * H, S, hd), dtype=torch.float16, device=dev)
    t_att = timed(lambda: blk.fa.ForwardEx(q3[0].codes.data_ptr(), q3[1].codes.data_ptr(), q3[2].codes.data_ptr(), o.data_ptr(), 0,
                                           B * H, S, hd, 1, 0, 1 / math.sqrt(hd), 1.0, q3[0].scale_ptr, q3[1].scale_ptr, q3[2].scale_ptr, sh))
    fl_gemm = 2.0 * M * d * (3 * d + d + 3 * Fh)
    fl_att = 2.0 * B * H * S * S * hd
    kern = t_qkv + t_o + t_gu + t_dn + t_att
    print(f"block B={B} S={S} d={d} H={H} F={Fh}: total {total:.3f} ms; FP8 kernels {kern:.3f} ms "
          f"(qkv {t_qkv:.3f}, o {t_o:.3f}, gate+up {t_gu:.3f}, down {t_dn:.3f}, attention {t_att:.3f}); fused glue+quantise {total - kern:.3f} ms; "
          f"same block with torch glue and separate quantiser calls {total_unfused:.3f} ms")
    print(f"GEMM {fl_gemm / (t_qkv + t_o + t_gu + t_dn) / 1e9:.0f} TFLOPS over {fl_gemm / 1e12:.2f} TFLOP; "
          f"attention (causal) {fl_att / t_att / 1e9:.0f} TFLOPS; whole block {(fl_gemm + fl_att) / total / 1e9:.0f} TFLOPS")
    blk.close()


if __name__ == "__main__":
    _main()
