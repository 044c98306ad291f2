"""Workloads that the framework's performance is judged by.

Each case is one pass through the public entry points as a program that serves (or evaluates) a quantised model makes it:
attention on e4m3 codes (`FAContext.ForwardEx`), GEMMs on e4m3 codes (`FP8GEMMScaled`), a linear layer on fp32 activations
(`nn.FP8Linear`), one decoder block over a prompt (`nn.FP8DecoderBlock`), the same block for one new token per sequence
(`decode_step`), and the attention part of a decode step with grouped-query heads on a paged cache (`DecodeRopeAppend` +
`FAContext.Decode`).  `listed()` holds the named cases, `draw()` gives more of the same ranges, `prepare()` makes what the
program has in hand before the call, `run()` is the pass, `work()` its unavoidable bytes and operations and `tolerance()`
how far another correct implementation may be off.
"""
import math

import torch

from goml_b200 import block_glue as BG, fa_forward as F, fp8_gemm as G, nn

DEV = "cuda"
CODE_STD = 80.0   # N(0,1) data quantised with scale = amax/448 has codes of about this spread (amax is 5 to 6 sigma)
THETA = 10000.0

#: (d_model, heads, feed-forward width) of the blocks: the full-size block, a half-width one of head dim 128 and one of 64
BLOCKS = [(4096, 32, 11008), (2048, 16, 5504), (2048, 32, 5632)]


def listed():
    full = dict(d=4096, heads=32, ffn=11008)
    return [
        # one short sequence, head dim 64, every key visible: the smallest call, where launches and host work count
        dict(name="attn_tiny", kind="attention", bh=4, s=256, hd=64, causal=False, window=0, lse=False),
        # sliding-window attention of a small model on a length that is no multiple of anything, LSE kept (training forward)
        dict(name="attn_window_hd64", kind="attention", bh=64, s=3000, hd=64, causal=True, window=512, lse=True),
        # causal prompt attention of eight 2048-token sequences with 32 heads of 128
        dict(name="attn_prefill", kind="attention", bh=256, s=2048, hd=128, causal=True, window=0, lse=False),
        # long-sequence forward with LSE, the largest attention call
        dict(name="attn_long", kind="attention", bh=128, s=8192, hd=128, causal=False, window=0, lse=True),
        # a projection for 16 tokens: reads the weight once
        dict(name="gemm_skinny", kind="gemm", m=16, n=8192, k=8192, out="fp16"),
        # the square GEMM
        dict(name="gemm_square", kind="gemm", m=8192, n=8192, k=8192, out="bf16"),
        # one linear layer on fp32 activations of a ragged batch of tokens: quantise, then multiply
        dict(name="linear_ragged", kind="linear", rows=3001, k=4096, n=11008),
        # a short prompt of one user through a block, K and V kept for decoding
        dict(name="prefill_short", kind="prefill", batch=1, s=173, **full),
        # eight full prompts through a block, K and V kept for decoding
        dict(name="prefill_full", kind="prefill", batch=8, s=2048, **full),
        # one user's next token
        dict(name="decode_one", kind="decode", batch=1, s=1000, **full),
        # the next token of 64 users whose contexts are 2048 to 4096 tokens long
        dict(name="decode_batch", kind="decode", batch=64, s=4096, **full),
        # attention part of a decode step on a paged cache, four query heads per kv head
        dict(name="decode_gqa_paged", kind="paged", batch=24, q_heads=32, kv_heads=8, hd=128, s=6000, page=128),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attention", "gemm", "linear", "prefill", "decode", "paged"])
    if kind == "attention":
        hd = rng.choice([64, 128])
        causal = rng.random() < 0.6
        s = _log(rng, 128, 8192)
        most = min(256, int(2.0e12 / (4.0 * s * s * hd)))
        window = rng.randint(64, s) if causal and rng.random() < 0.25 else 0
        return dict(kind=kind, bh=_log(rng, 4, max(5, most)), s=s, hd=hd, causal=causal, window=window, lse=rng.random() < 0.5)
    if kind == "gemm":
        n, k = _log(rng, 1024, 8192), 16 * _log(rng, 64, 512)
        if rng.random() < 0.7:
            n = n // 8 * 8
        return dict(kind=kind, m=_log(rng, 1, 8192), n=n, k=k, out=rng.choice(["fp16", "bf16"]))
    if kind == "linear":
        return dict(kind=kind, rows=_log(rng, 1, 8192), k=16 * _log(rng, 64, 512), n=8 * _log(rng, 128, 1376))
    if kind == "paged":
        hd, page = rng.choice([64, 128, 128]), rng.choice([64, 128, 256])
        kv, s = rng.choice([4, 8]), _log(rng, 200, 8192)
        most = min(64, int(1.0e9 / (2.0 * kv * hd * s)))
        return dict(kind=kind, batch=_log(rng, 1, max(2, most)), q_heads=kv * rng.choice([4, 8]), kv_heads=kv, hd=hd, s=s, page=page)
    d, heads, ffn = rng.choice(BLOCKS)
    if kind == "prefill":
        s = _log(rng, 32, 2048)
        return dict(kind=kind, batch=_log(rng, 1, max(2, min(16, 8192 // s))), s=s, d=d, heads=heads, ffn=ffn)
    s = _log(rng, 128, 8192)
    return dict(kind=kind, batch=_log(rng, 1, max(2, min(96, int(1.5e9 / (2.0 * d * s))))), s=s, d=d, heads=heads, ffn=ffn)


# ------------------------------------------------------------------------------------------------ what a case consists of
def _lengths(c):
    """Cached keys of each sequence: s, and less in equal steps down to half of that."""
    return [c["s"] - i * c["s"] // (2 * c["batch"]) for i in range(c["batch"])]


def _out_type(c):
    return (torch.float16, G.OutFP16) if c["out"] == "fp16" else (torch.bfloat16, G.OutBF16)


def _pairs(c):
    """(query, key) pairs one head's attention looks at."""
    s, w = c["s"], c["window"]
    if not c["causal"]:
        return s * s
    if w == 0 or w >= s:
        return s * (s + 1) / 2
    return w * (w + 1) / 2 + (s - w) * w


def work(c):
    if c["kind"] == "attention":
        rows = c["bh"] * c["s"]
        return {"bytes": rows * (3.0 * c["hd"] + 2 * c["hd"] + (4 if c["lse"] else 0)), "flops": 4.0 * c["bh"] * c["hd"] * _pairs(c)}
    if c["kind"] == "gemm":
        m, n, k = c["m"], c["n"], c["k"]
        return {"bytes": 1.0 * m * k + n * k + 2.0 * m * n, "flops": 2.0 * m * n * k}
    if c["kind"] == "linear":
        m, n, k = c["rows"], c["n"], c["k"]
        return {"bytes": 4.0 * m * k + n * k + 2.0 * m * n, "flops": 2.0 * m * n * k}
    if c["kind"] == "paged":
        keys = sum(_lengths(c)) + c["batch"]
        return {"bytes": 2.0 * keys * c["kv_heads"] * c["hd"] + c["batch"] * (2.0 * (c["q_heads"] + 2 * c["kv_heads"]) + 2 * c["q_heads"]) * c["hd"],
                "flops": 4.0 * keys * c["q_heads"] * c["hd"]}
    d, ffn, B = c["d"], c["ffn"], c["batch"]
    weights = 4.0 * d * d + 3.0 * d * ffn
    if c["kind"] == "prefill":
        t = B * c["s"]
        return {"bytes": weights + 8.0 * t * d + 2.0 * t * d, "flops": 2.0 * t * weights + 4.0 * B * d * c["s"] * (c["s"] + 1) / 2}
    keys = sum(_lengths(c)) + B
    return {"bytes": weights + 8.0 * B * d + 2.0 * keys * d, "flops": 2.0 * B * weights + 4.0 * keys * d}


def tolerance(c):
    if c["kind"] == "attention" or c["kind"] == "paged":
        return {"rel": 2e-3, "max": 2e-2, "differ": 0.0}          # fp16 output; codes and lengths are exact
    if c["kind"] == "gemm":
        return {"rel": 2e-3 if c["out"] == "fp16" else 5e-3}      # fp32 accumulation, one rounding to the output type
    if c["kind"] == "linear":
        return {"rel": 5e-3}                                      # exact codes, fp32 accumulation, bf16 output
    # a block re-quantises between its stages: a last-bit difference becomes an isolated neighbouring e4m3 code
    return {"rel": 1e-2, "max": 0.4, "differ": 5e-3}


# --------------------------------------------------------------------------------------------------------------- the pass
_CTX = None


def _context():
    """One attention context per process and GPU, as a program keeps it."""
    global _CTX
    if _CTX is None:
        _CTX = F.FACreate()
    return _CTX


def _codes(g, *shape):
    """e4m3 codes of N(0,1) data; the scale that belongs to them is 1 / CODE_STD."""
    out = torch.empty(shape, dtype=torch.uint8, device=DEV)
    flat = out.view(-1)
    step = 1 << 27
    for i in range(0, flat.numel(), step):
        part = flat[i:i + step]
        x = torch.randn(part.numel(), generator=g, device=DEV).mul_(CODE_STD).clamp_(-448, 448)
        part.copy_(x.to(torch.float8_e4m3fn).view(torch.uint8))
    return out


def _block(c, g):
    rn = lambda *shape: torch.randn(*shape, generator=g, device=DEV).mul_(0.02)
    d, ffn = c["d"], c["ffn"]
    gain = lambda: 1.0 + 5.0 * rn(d)
    return nn.FP8DecoderBlock(d, c["heads"], ffn, rn(3 * d, d), rn(d, d), rn(2 * ffn, d), rn(d, ffn), gain(), gain())


def prepare(c, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    st = {"case": c, "stream": torch.cuda.current_stream().cuda_stream}
    if c["kind"] == "attention":
        shape = (c["bh"], c["s"], c["hd"])
        st["qkv"] = [_codes(g, *shape) for _ in range(3)]
        st["scales"] = torch.full((3,), 1.0 / CODE_STD, device=DEV)
        st["o"] = torch.empty(shape, dtype=torch.float16, device=DEV)
        st["lse"] = torch.empty(shape[:2], dtype=torch.float32, device=DEV) if c["lse"] else None
        st["ctx"] = _context()
    elif c["kind"] == "gemm":
        st["a"], st["b"] = _codes(g, c["m"], c["k"]), _codes(g, c["n"], c["k"])
        st["scales"] = torch.full((2,), 1.0 / CODE_STD, device=DEV)
        st["c"] = torch.empty((c["m"], c["n"]), dtype=_out_type(c)[0], device=DEV)
    elif c["kind"] == "linear":
        st["layer"] = nn.FP8Linear(torch.randn(c["n"], c["k"], generator=g, device=DEV).mul_(0.02))
        st["x"] = torch.randn(c["rows"], c["k"], generator=g, device=DEV)
    elif c["kind"] == "paged":
        B, hq, hkv, hd, page = c["batch"], c["q_heads"], c["kv_heads"], c["hd"], c["page"]
        per_seq = (c["s"] + 1 + page - 1) // page
        st["per_seq"], st["pages"] = per_seq, B * per_seq
        st["k"], st["v"] = _codes(g, B * per_seq, hkv, page, hd), _codes(g, B * per_seq, hkv, page, hd)
        st["table"] = torch.randperm(B * per_seq, generator=g, device=DEV).to(torch.int32).view(B, per_seq)
        order = torch.randperm(B, generator=g, device=DEV)
        st["lens"] = torch.tensor(_lengths(c), dtype=torch.int32, device=DEV)[order]
        st["lens_next"] = torch.empty_like(st["lens"])
        st["rows"] = c["s"] + 1
        st["cos"] = torch.empty((st["rows"], hd // 2), dtype=torch.float32, device=DEV)
        st["sin"] = torch.empty_like(st["cos"])
        BG.RopeTable(st["cos"].data_ptr(), st["sin"].data_ptr(), st["rows"], hd, THETA, st["stream"])
        st["qkv"] = torch.randn(B, (hq + 2 * hkv) * hd, generator=g, device=DEV).to(torch.bfloat16)
        st["q"] = torch.empty((B, hq, hd), dtype=torch.uint8, device=DEV)
        st["qs"] = torch.empty(2, dtype=torch.float32, device=DEV)
        st["kv_scales"] = torch.full((2,), 1.0 / CODE_STD, device=DEV)
        st["o"] = torch.empty((B, hq, hd), dtype=torch.float16, device=DEV)
        st["ctx"] = _context()
    else:
        st["block"] = _block(c, g)
        B, hd = c["batch"], c["d"] // c["heads"]
        if c["kind"] == "prefill":
            st["x"] = torch.randn(B * c["s"], c["d"], generator=g, device=DEV)
            st["cache"] = nn.FP8KVCache(B, c["heads"], c["s"] + 64, hd)   # room for the answer
        else:
            st["x"] = torch.randn(B, c["d"], generator=g, device=DEV)
            cache = nn.FP8KVCache(B, c["heads"], c["s"] + 64, hd)
            cache.k, cache.v = _codes(g, *cache.k.shape), _codes(g, *cache.v.shape)
            cache.scales.fill_(1.0 / CODE_STD)
            order = torch.randperm(B, generator=g, device=DEV)
            st["lens"] = torch.tensor(_lengths(c), dtype=torch.int32, device=DEV)[order]
            st["cache"] = cache
    return st


def run(st):
    c, stream = st["case"], st["stream"]
    if c["kind"] == "attention":
        q, k, v = st["qkv"]
        s = st["scales"].data_ptr()
        lse = st["lse"]
        st["ctx"].ForwardEx(q.data_ptr(), k.data_ptr(), v.data_ptr(), st["o"].data_ptr(), 0 if lse is None else lse.data_ptr(),
                            c["bh"], c["s"], c["hd"], int(c["causal"]), c["window"], 1.0 / math.sqrt(c["hd"]), 1.0, s, s + 4, s + 8, stream)
        return st["o"] if lse is None else (st["o"], lse)
    if c["kind"] == "gemm":
        s = st["scales"].data_ptr()
        G.FP8GEMMScaled(c["m"], c["n"], c["k"], st["a"].data_ptr(), st["b"].data_ptr(), st["c"].data_ptr(), 1.0, s, s + 4, _out_type(c)[1], stream)
        return st["c"]
    if c["kind"] == "linear":
        return st["layer"](st["x"])
    if c["kind"] == "paged":
        B, hq, hkv, hd = c["batch"], c["q_heads"], c["kv_heads"], c["hd"]
        qs, kvs = st["qs"].data_ptr(), st["kv_scales"].data_ptr()
        BG.DecodeRopeAppend(st["qkv"].data_ptr(), st["cos"].data_ptr(), st["sin"].data_ptr(), st["lens"].data_ptr(), st["q"].data_ptr(), qs, qs + 4,
                            st["k"].data_ptr(), st["v"].data_ptr(), kvs, kvs + 4, B, hq, hkv, hd, 0, st["rows"],
                            seq_lens_out=st["lens_next"].data_ptr(), block_table=st["table"].data_ptr(), page_size=c["page"],
                            max_pages_per_seq=st["per_seq"], num_pages=st["pages"], stream=stream)
        st["ctx"].Decode(st["q"].data_ptr(), st["k"].data_ptr(), st["v"].data_ptr(), st["o"].data_ptr(), 0, st["lens_next"].data_ptr(), B, hq, hkv, hd,
                         0, 0, 1.0 / math.sqrt(hd), 1.0, qs, kvs, kvs + 4, stream, block_table=st["table"].data_ptr(), page_size=c["page"],
                         max_pages_per_seq=st["per_seq"], num_pages=st["pages"])
        return st["o"], st["q"], st["qs"], st["k"], st["v"], st["lens_next"]
    cache = st["cache"]
    if c["kind"] == "prefill":
        y = st["block"](st["x"], c["batch"], c["s"], cache)
        return y, cache.k, cache.v, cache.scales, cache.lens
    cache.lens.copy_(st["lens"])   # a server hands every step the lengths of the sequences it has scheduled
    y = st["block"].decode_step(st["x"], cache)
    return y, cache.k, cache.v, cache.lens
