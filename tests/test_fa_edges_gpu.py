"""Attention forward where masks cut key blocks: every 32-key chunk of a block is masked, left alone or skipped per warp."""
import math

import numpy as np
import pytest

import oracle as O
from tests.gpu_util import run_attention

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
