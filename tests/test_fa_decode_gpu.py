"""Decode step (one new token per sequence, FP8 KV cache, grouped-query heads) against the fp64 restatement.

Tolerance: the stated bar of the path (max-abs <= 2e-2, mean relative <= 1e-2 on the fp16 output; LSE within 5e-3).
The reference has no implementation of this step (design notes only), so there is no golden vector to pin:
parity unpinned; the restatement is the single-row case of the attention restatement the prefill tests use, and
one test below checks the decode kernel against the prefill kernel's last row on the same cache.
"""
import math

import numpy as np
import pytest
import torch

import oracle as O
from oracle import glue

pytestmark = pytest.mark.gpu


def run_decode(ctx, q, kc, vc, seq_lens, scale, v_descale=1.0, s_max=None, uniform_len=None):
    B, Hq, D = q.shape
    Hkv, Smax = kc.shape[1], kc.shape[2]
    qd, kd, vd = (torch.from_numpy(np.ascontiguousarray(t)).cuda() for t in (q, kc, vc))
    o = torch.full((B, Hq, D), float("nan"), dtype=torch.float16, device="cuda")
    lse = torch.full((B, Hq), float("nan"), dtype=torch.float32, device="cuda")
    sl = None if uniform_len is not None else torch.from_numpy(np.asarray(seq_lens, np.int32)).cuda()
    ctx.Decode(qd.data_ptr(), kd.data_ptr(), vd.data_ptr(), o.data_ptr(), lse.data_ptr(), 0 if sl is None else sl.data_ptr(),
               B, Hq, Hkv, D, Smax, uniform_len or 0, scale, v_descale)
    torch.cuda.synchronize()
    ctx.DeviceStatus()
    return o.double().cpu().numpy(), lse.double().cpu().numpy()


def make_case(name, B, Hq, Hkv, Smax, D):
    qf = O.seeded_normal("q", (B, Hq, D), config=name)
    kf = O.seeded_normal("k", (B, Hkv, Smax, D), config=name)
    vf = O.seeded_normal("v", (B, Hkv, Smax, D), config=name)
    (q, sq, _), (k, sk, _), (v, sv, _) = (O.quantize_f32(t) for t in (qf, kf, vf))
    return q, k, v, float(sq), float(sk), float(sv)


@pytest.mark.parametrize("B,Hq,Hkv,Smax,D", [(2, 8, 2, 300, 128), (3, 4, 4, 64, 64), (1, 16, 1, 1000, 128), (5, 12, 4, 129, 64),
                                             (2, 32, 8, 2048, 128)])
def test_decode_matches_restatement(cuda, built_libs, fa_ctx, B, Hq, Hkv, Smax, D):
    name = f"decode{B}_{Hq}_{Hkv}_{Smax}_{D}"
    q, k, v, sq, sk, sv = make_case(name, B, Hq, Hkv, Smax, D)
    rng = np.random.default_rng(B * 131 + Smax)
    seq_lens = rng.integers(1, Smax + 1, size=B)
    seq_lens[0] = Smax                       # one full-length sequence
    scale = sq * sk / math.sqrt(D)
    got, lse = run_decode(fa_ctx, q, k, v, seq_lens, scale, sv)
    ref, rl = glue.decode_attention_f64(q, k, v, seq_lens, scale, sv)
    assert np.isfinite(got).all()
    maxabs, meanrel = O.error_stats(got, ref)
    assert maxabs <= 2e-2 and meanrel <= 1e-2, (maxabs, meanrel)
    assert np.abs(lse - rl).max() <= 5e-3


def test_uniform_length_and_empty_sequences(cuda, built_libs, fa_ctx):
    B, Hq, Hkv, Smax, D = 3, 8, 2, 200, 128
    q, k, v, sq, sk, sv = make_case("decode-uniform", B, Hq, Hkv, Smax, D)
    scale = sq * sk / math.sqrt(D)
    got, lse = run_decode(fa_ctx, q, k, v, None, scale, sv, uniform_len=77)
    ref, rl = glue.decode_attention_f64(q, k, v, [77] * B, scale, sv)
    maxabs, meanrel = O.error_stats(got, ref)
    assert maxabs <= 2e-2 and meanrel <= 1e-2 and np.abs(lse - rl).max() <= 5e-3
    # a sequence with no visible key: O = 0, LSE = -inf; lengths beyond s_max are clamped
    got, lse = run_decode(fa_ctx, q, k, v, [0, 50, 10 ** 6], scale, sv)
    ref, rl = glue.decode_attention_f64(q, k, v, [0, 50, Smax], scale, sv)
    assert np.all(got[0] == 0) and np.all(np.isneginf(lse[0]))
    maxabs, meanrel = O.error_stats(got[1:], ref[1:])
    assert maxabs <= 2e-2 and meanrel <= 1e-2 and np.abs(lse[1:] - rl[1:]).max() <= 5e-3


def test_decode_equals_last_row_of_prefill(cuda, built_libs, fa_ctx):
    # the same cache through the prefill kernel (causal): its last query row is the decode step's answer
    from tests.gpu_util import run_attention
    BH, S, D = 4, 320, 128
    q, k, v, sq, sk, sv = make_case("decode-vs-prefill", BH, 1, 1, S, D)      # q: [BH, 1, D] (one query head per kv head)
    qfull = np.zeros((BH, S, D), np.uint8)
    qfull[:, S - 1] = q[:, 0]
    scale = sq * sk / math.sqrt(D)
    o_pre, lse_pre = run_attention(fa_ctx, qfull, k[:, 0], v[:, 0], causal=1, scale=scale, v_descale=sv, entry="ex")
    got, lse = run_decode(fa_ctx, q, k, v, [S] * BH, scale, sv)
    assert np.abs(got[:, 0] - o_pre[:, S - 1]).max() <= 2e-3
    assert np.abs(lse[:, 0] - lse_pre[:, S - 1]).max() <= 1e-4


def test_rejects_bad_arguments(cuda, built_libs, fa_ctx):
    from goml_b200 import fa_forward as F
    buf = torch.zeros(1 << 16, dtype=torch.uint8, device="cuda")
    p = buf.data_ptr()
    for args, code in [((p, p, p, p, 0, 0, 1, 6, 4, 128, 64, 64, 1.0), F.FA_ERR_UNSUPPORTED_SHAPE),    # 6 % 4 != 0
                       ((p, p, p, p, 0, 0, 1, 32, 1, 128, 64, 64, 1.0), F.FA_ERR_UNSUPPORTED_SHAPE),   # 32 query heads per kv head
                       ((p, p, p, p, 0, 0, 1, 8, 2, 96, 64, 64, 1.0), F.FA_ERR_UNSUPPORTED_HD),
                       ((p, p, p, p, 0, 0, 1, 8, 2, 128, 64, 65, 1.0), F.FA_ERR_INVALID_ARG),          # seq_len > s_max
                       ((p, 0, p, p, 0, 0, 1, 8, 2, 128, 64, 64, 1.0), F.FA_ERR_INVALID_ARG)]:
        with pytest.raises(F.FAError) as e:
            fa_ctx.Decode(*args)
        assert e.value.status == code, (args, e.value.status)


def to_pages(cache, page, rng, spare=3):
    """Contiguous [B, Hkv, S, D] cache -> (pool [P, Hkv, page, D], table [B, S/page]) with the pages of every
    sequence scattered over a pool that also holds `spare` unused pages full of NaN codes."""
    B, Hkv, S, D = cache.shape
    per_seq = S // page
    P = B * per_seq + spare
    pool = np.full((P, Hkv, page, D), 0x7F, np.uint8)
    table = rng.permutation(P)[:B * per_seq].astype(np.int32).reshape(B, per_seq)
    for b in range(B):
        for j in range(per_seq):
            pool[table[b, j]] = cache[b, :, j * page:(j + 1) * page]
    return pool, table


@pytest.mark.parametrize("B,Hq,Hkv,S,D,page", [(3, 8, 2, 512, 128, 64), (2, 16, 4, 1024, 64, 256), (4, 8, 8, 384, 128, 128),
                                               (2, 32, 8, 4096, 128, 512)])
def test_paged_cache_equals_contiguous_cache(cuda, built_libs, fa_ctx, B, Hq, Hkv, S, D, page):
    # the same keys and values behind a block table: same split of the key range, same arithmetic -> identical bits
    name = f"paged{B}_{Hq}_{Hkv}_{S}_{D}_{page}"
    q, k, v, sq, sk, sv = make_case(name, B, Hq, Hkv, S, D)
    rng = np.random.default_rng(S + page)
    seq_lens = rng.integers(1, S + 1, size=B).astype(np.int32)
    seq_lens[0] = S
    scale = sq * sk / math.sqrt(D)
    want, want_lse = run_decode(fa_ctx, q, k, v, seq_lens, scale, sv)
    ref, rl = glue.decode_attention_f64(q, k, v, seq_lens, scale, sv)
    kp, table = to_pages(k, page, rng)
    # one table serves both pools, so V is laid out with K's table
    vp = np.full_like(kp, 0xFF)
    for b in range(B):
        for j in range(S // page):
            vp[table[b, j]] = v[b, :, j * page:(j + 1) * page]
    table_dev = table.copy()
    for b in range(B):                                    # entries past a sequence's pages are never read: poison them
        table_dev[b, (int(seq_lens[b]) + page - 1) // page:] = -12345
    qd, kd, vd, td = (torch.from_numpy(np.ascontiguousarray(t)).cuda() for t in (q, kp, vp, table_dev))
    sl = torch.from_numpy(seq_lens).cuda()
    o = torch.full((B, Hq, D), float("nan"), dtype=torch.float16, device="cuda")
    lse = torch.full((B, Hq), float("nan"), dtype=torch.float32, device="cuda")
    fa_ctx.Decode(qd.data_ptr(), kd.data_ptr(), vd.data_ptr(), o.data_ptr(), lse.data_ptr(), sl.data_ptr(), B, Hq, Hkv, D, 0, 0,
                  scale, sv, block_table=td.data_ptr(), page_size=page, max_pages_per_seq=S // page, num_pages=kp.shape[0])
    torch.cuda.synchronize()
    fa_ctx.DeviceStatus()
    got, got_lse = o.double().cpu().numpy(), lse.double().cpu().numpy()
    assert np.array_equal(got, want) and np.array_equal(got_lse, want_lse)
    maxabs, meanrel = O.error_stats(got, ref)
    assert maxabs <= 2e-2 and meanrel <= 1e-2 and np.abs(got_lse - rl).max() <= 5e-3


def test_bytes_past_the_sequence_length_are_never_used(cuda, built_libs, fa_ctx):
    # a cache that was allocated and not cleared holds arbitrary bytes past each sequence's end, NaN codes included:
    # the result must be bit-identical to the one over a clean cache
    B, Hq, Hkv, S, D = 4, 8, 2, 300, 128
    q, k, v, sq, sk, sv = make_case("decode-stale", B, Hq, Hkv, S, D)
    seq_lens = np.array([1, 63, 130, 299], np.int32)
    scale = sq * sk / math.sqrt(D)
    want, want_lse = run_decode(fa_ctx, q, k, v, seq_lens, scale, sv)
    k2, v2 = k.copy(), v.copy()
    for b, n in enumerate(seq_lens):
        k2[b, :, n:] = 0x7F
        v2[b, :, n:] = 0xFF
    got, got_lse = run_decode(fa_ctx, q, k2, v2, seq_lens, scale, sv)
    assert np.isfinite(got).all()
    assert np.array_equal(got, want) and np.array_equal(got_lse, want_lse)


def test_paged_rejects_bad_page_size(cuda, built_libs, fa_ctx):
    from goml_b200 import fa_forward as F
    buf = torch.zeros(1 << 16, dtype=torch.uint8, device="cuda")
    p = buf.data_ptr()
    for kw in (dict(page_size=48, max_pages_per_seq=2, num_pages=4), dict(page_size=64, max_pages_per_seq=0, num_pages=4),
               dict(page_size=64, max_pages_per_seq=2, num_pages=0)):
        with pytest.raises(F.FAError) as e:
            fa_ctx.Decode(p, p, p, p, 0, 0, 1, 8, 2, 128, 0, 64, 1.0, block_table=p, **kw)
        assert e.value.status == F.FA_ERR_INVALID_ARG


@pytest.mark.parametrize("B,Hq,Hkv,Smax,D,lens", [
    (150, 2, 1, 70, 128, "ramp"),        # more sequences than a warp keeps lengths for, empty ones among them
    (40, 9, 1, 130, 64, "ramp"),         # nine query heads per kv head: two column tiles, the second nearly empty
    (1, 3, 1, 20000, 128, "full"),       # one pair cut into hundreds of pieces (several batches of the merge)
    (1, 16, 1, 9000, 64, "full"),
    (2, 8, 8, 65, 128, "full"),          # fewer chunks than CTAs: every chunk is a piece, a one-key second chunk
    (7, 4, 2, 1500, 128, "one long"),    # one long sequence among very short ones
    (25, 32, 32, 200, 128, "ramp"),      # one query head per kv head, more pairs than CTAs: each pair cut at most once
    (23, 30, 30, 1100, 64, "one long"),
    (40, 32, 32, 2050, 128, "ramp"),     # a CTA per pair: wide steps, empty sequences among them, one key in the last chunk
    (70, 16, 16, 2047, 128, "one long"),
    (19, 32, 32, 2049, 64, "ramp"),
    (60, 32, 8, 900, 128, "ramp"),       # groups with a CTA per pair
    (180, 8, 8, 65, 64, "one long"),
    (200, 32, 8, 130, 64, "ramp"),
    (61, 64, 4, 1025, 64, "one long"),   # two column tiles, a CTA per pair: wide and narrow steps
    (70, 40, 4, 500, 128, "ramp"),
    (300, 9, 1, 70, 64, "ramp"),
    (130, 48, 4, 600, 128, "one long"),
])
def test_decode_work_split(cuda, built_libs, fa_ctx, B, Hq, Hkv, Smax, D, lens):
    # the key range is cut at chunk borders wherever the pieces of the work line end, whatever the lengths are
    name = f"decode-split{B}_{Hq}_{Hkv}_{Smax}_{D}"
    q, k, v, sq, sk, sv = make_case(name, B, Hq, Hkv, Smax, D)
    seq_lens = {"ramp": np.arange(B) * Smax // B, "full": np.full(B, Smax), "one long": np.where(np.arange(B) == 3, Smax, 1 + np.arange(B))}[lens]
    scale = sq * sk / math.sqrt(D)
    got, lse = run_decode(fa_ctx, q, k, v, seq_lens, scale, sv)
    again, lse2 = run_decode(fa_ctx, q, k, v, seq_lens, scale, sv)
    ref, rl = glue.decode_attention_f64(q, k, v, seq_lens, scale, sv)
    assert np.array_equal(got, again) and np.array_equal(lse, lse2)      # merged in a fixed order
    some = seq_lens > 0
    assert np.all(got[~some] == 0) and np.all(np.isneginf(lse[~some]))
    maxabs, meanrel = O.error_stats(got[some], ref[some])
    assert maxabs <= 2e-2 and meanrel <= 1e-2, (maxabs, meanrel)
    assert np.abs(lse[some] - rl[some]).max() <= 5e-3


@pytest.mark.parametrize("B,Hq,Hkv,D", [(256, 1, 1, 64), (64, 8, 4, 128), (128, 10, 2, 64), (3, 2, 2, 64)])
def test_capacity_far_above_what_is_held(cuda, built_libs, fa_ctx, B, Hq, Hkv, D):
    # 2^30 rows a sequence in the block table (2^24 chunks of 64 keys: with 256 pairs more than an int counts), few of them
    # held; unused entries name no page
    page, max_pages, held = 65536, 16384, 3
    name = f"decode-capacity{B}_{Hq}_{Hkv}_{D}"
    q, k, v, sq, sk, sv = make_case(name, B, Hq, Hkv, 150, D)
    seq_lens = np.arange(B) % 151
    kd, vd = (torch.zeros(held, Hkv, page, D, dtype=torch.uint8, device="cuda") for _ in range(2))
    for i in range(held):    # sequence b lives in page b % 3: the content of the first three sequences
        kd[i, :, :150], vd[i, :, :150] = torch.from_numpy(k[i % B]).cuda(), torch.from_numpy(v[i % B]).cuda()
    table = torch.full((B, max_pages), -1, dtype=torch.int32, device="cuda")
    table[:, 0] = torch.arange(B, device="cuda") % held
    scale = sq * sk / math.sqrt(D)
    qd, sl = torch.from_numpy(q).cuda(), torch.from_numpy(seq_lens.astype(np.int32)).cuda()
    o = torch.full((B, Hq, D), float("nan"), dtype=torch.float16, device="cuda")
    lse = torch.full((B, Hq), float("nan"), dtype=torch.float32, device="cuda")
    fa_ctx.Decode(qd.data_ptr(), kd.data_ptr(), vd.data_ptr(), o.data_ptr(), lse.data_ptr(), sl.data_ptr(), B, Hq, Hkv, D, 0, 0, scale, sv,
                  block_table=table.data_ptr(), page_size=page, max_pages_per_seq=max_pages, num_pages=held)
    torch.cuda.synchronize()
    fa_ctx.DeviceStatus()
    src = np.arange(B) % held % B
    ref, rl = glue.decode_attention_f64(q, k[src], v[src], seq_lens, scale, sv)
    some = seq_lens > 0
    got, glse = o.double().cpu().numpy(), lse.double().cpu().numpy()
    assert np.all(got[~some] == 0) and np.all(np.isneginf(glse[~some]))
    maxabs, meanrel = O.error_stats(got[some], ref[some])
    assert maxabs <= 2e-2 and meanrel <= 1e-2, (maxabs, meanrel)
    assert np.abs(glse[some] - rl[some]).max() <= 5e-3


@pytest.mark.parametrize("B,H,Smax,D,cluster", [(1, 16, 100, 64, True), (9, 32, 200, 64, True), (5, 16, 900, 64, True), (3, 16, 500, 128, True), (1, 32, 1064, 128, True),
                                                (1, 16, 2000, 64, True), (1, 32, 3000, 128, False), (1, 16, 2500, 64, False), (1, 9, 4100, 128, False)])
def test_splits_in_clusters_and_in_the_workspace(cuda, built_libs, fa_ctx, B, H, Smax, D, cluster):
    # clusters of 2 to 16 CTAs with runs of one to three splits, and up to 64 splits that meet in the workspace: whole and part chunks, fewer than CTAs, none; the
    # paged cache has the same bits
    from tests.gpu_util import kernels
    q, k, v, sq, sk, sv = make_case(f"cluster{B}_{H}_{Smax}_{D}", B, H, H, Smax, D)
    rng = np.random.default_rng(Smax)
    scale = sq * sk / math.sqrt(D)
    sets = [rng.integers(1, Smax + 1, size=B) for _ in range(2)] + [np.full(B, n) for n in (Smax, 1, 64, 65, 0)]
    per_seq = -(-Smax // 64)
    pad = np.zeros((B, H, per_seq * 64, D), np.uint8)
    table = rng.permutation(B * per_seq).reshape(B, per_seq).astype(np.int32)
    pools = []
    for cache in (k, v):
        pad[:, :, :Smax] = cache
        pool = np.empty((B * per_seq, H, 64, D), np.uint8)
        pool[table.ravel()] = pad.reshape(B, H, per_seq, 64, D).transpose(0, 2, 1, 3, 4).reshape(-1, H, 64, D)
        pools.append(torch.from_numpy(pool).cuda())
    qd, td = torch.from_numpy(q).cuda(), torch.from_numpy(table).cuda()
    for n, lens in enumerate(sets):
        got, lse = run_decode(fa_ctx, q, k, v, lens, scale, sv)
        o = torch.full((B, H, D), float("nan"), dtype=torch.float16, device="cuda")
        ld = torch.from_numpy(np.asarray(lens, np.int32)).cuda()
        call = lambda: fa_ctx.Decode(qd.data_ptr(), pools[0].data_ptr(), pools[1].data_ptr(), o.data_ptr(), 0, ld.data_ptr(), B, H, H, D, 0, 0, scale, sv,
                                     stream=torch.cuda.current_stream().cuda_stream, block_table=td.data_ptr(), page_size=64, max_pages_per_seq=per_seq, num_pages=B * per_seq)
        call()
        torch.cuda.synchronize()
        assert np.array_equal(o.double().cpu().numpy(), got)
        if n == 0:
            assert len(kernels(call)) == (1 if cluster else 2)   # the workspace's words are cleared by another
        if not lens.any():
            assert (got == 0).all() and np.isneginf(lse).all()
            continue
        ref, rl = glue.decode_attention_f64(q, k, v, lens, scale, sv)
        maxabs, meanrel = O.error_stats(got, ref)
        assert maxabs <= 2e-2 and meanrel <= 1e-2, (lens, maxabs, meanrel)
        assert np.abs(lse - rl).max() <= 5e-3


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,H,Smax,many", [(1, 8, 128, False), (1, 8, 512, False), (1, 8, 513, True), (2, 7, 575, True), (2, 7, 500, False), (3, 2, 2500, True), (1, 1, 4200, True)])
def test_few_and_many_pieces_in_the_workspace(cuda, built_libs, fa_ctx, B, H, Smax, D, many):
    # up to eight pieces of a pair are taken up by one group of threads, more by all of the block's, in a kernel of its own
    from tests.gpu_util import kernels
    x = torch.zeros(B * H * Smax * D, dtype=torch.uint8, device="cuda")
    o = torch.empty(B, H, D, dtype=torch.float16, device="cuda")
    names = kernels(lambda: fa_ctx.Decode(x.data_ptr(), x.data_ptr(), x.data_ptr(), o.data_ptr(), 0, 0, B, H, H, D, Smax, Smax, 1.0, 1.0, stream=torch.cuda.current_stream().cuda_stream))
    name, = (n for n in names if "fa_decode_kernel" in n)
    assert name.split("EvN")[0].endswith("Lb1ELb0EE" if many else "Lb0ELb0EE")
    test_splits_in_clusters_and_in_the_workspace(cuda, built_libs, fa_ctx, B, H, Smax, D, False)


@pytest.mark.parametrize("D,Smax", [(64, 2368), (64, 2000), (128, 2368), (128, 1800)])
def test_a_run_of_splits_is_rounded_as_splits_of_their_own(cuda, built_libs, fa_ctx, D, Smax):
    # A block of a cluster that takes two or three splits in turn starts a maximum for each: 16 heads are clusters, the first 15 of them meet in the workspace, and P
    # is rounded against the same maxima.  What differs is the order of fp32 sums, 2^-24 each against the 2^-11 of an fp16 result, so that few results fall
    # on the other side of a rounding; with one maximum for the run a model of the roundings differs in 24 to 34 % of them.
    from tests.gpu_util import kernels
    q, k, v, sq, sk, sv = make_case(f"runs{D}_{Smax}", 1, 16, 16, Smax, D)
    scale = sq * sk / math.sqrt(D)
    qd, kd, vd = (torch.from_numpy(t).cuda() for t in (q, k, v))
    o, ld = torch.empty(16, D, dtype=torch.float16, device="cuda"), torch.tensor([Smax], dtype=torch.int32, device="cuda")
    for heads, launches in ((16, 1), (15, 2)):   # the workspace's words are cleared by another
        assert len(kernels(lambda: fa_ctx.Decode(qd.data_ptr(), kd.data_ptr(), vd.data_ptr(), o.data_ptr(), 0, ld.data_ptr(), 1, heads, heads, D, Smax, 0, scale, sv,
                                                 stream=torch.cuda.current_stream().cuda_stream))) == launches
    for n in (Smax, Smax - 70, 1000, 200):
        (runs, lse), (own, own_lse) = (run_decode(fa_ctx, q[:, :h], k[:, :h], v[:, :h], [n], scale, sv) for h in (16, 15))
        assert (runs[:, :15] != own).mean() <= 0.02, (n, (runs[:, :15] != own).mean())
        assert np.abs(lse[:, :15] - own_lse).max() <= 1e-5


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,H,Smax,cluster", [(41, 4, 900, True), (42, 4, 900, False), (11, 16, 900, False), (46, 4, 130, True), (47, 4, 130, True), (74, 4, 500, True)])
def test_clusters_of_three_keep_clear_of_what_fits(cuda, built_libs, fa_ctx, D, B, H, Smax, cluster):
    # near the number that is resident at once they wait for one another; pairs of blocks do not (184 sequences and heads of three chunks are pairs), and all that there
    # is room for are taken
    from tests.gpu_util import kernels
    q, k, v, sq, sk, sv = make_case(f"threes{B}_{H}_{Smax}_{D}", B, H, H, Smax, D)
    scale = sq * sk / math.sqrt(D)
    qd, kd, vd = (torch.from_numpy(t).cuda() for t in (q, k, v))
    lens = np.random.default_rng(B).integers(1, Smax + 1, size=B)
    o, ld = torch.empty(B, H, D, dtype=torch.float16, device="cuda"), torch.from_numpy(lens.astype(np.int32)).cuda()
    names = kernels(lambda: fa_ctx.Decode(qd.data_ptr(), kd.data_ptr(), vd.data_ptr(), o.data_ptr(), 0, ld.data_ptr(), B, H, H, D, Smax, 0, scale, sv,
                                          stream=torch.cuda.current_stream().cuda_stream))
    assert len(names) == (1 if cluster else 2)   # the workspace's words are cleared by another
    got, lse = run_decode(fa_ctx, q, k, v, lens, scale, sv)
    ref, rl = glue.decode_attention_f64(q, k, v, lens, scale, sv)
    maxabs, meanrel = O.error_stats(got, ref)
    assert maxabs <= 2e-2 and meanrel <= 1e-2, (maxabs, meanrel)
    assert np.abs(lse - rl).max() <= 5e-3
