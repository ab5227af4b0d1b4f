"""Where the attention forward changes between one and two query tiles per CTA: both sides of each line, against the dense oracle."""
import math

import pytest
import torch

from archscale_b200.ops import backend
from archscale_b200.ops.attention import attention_ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,H,G,D,win", [
    (64, 100, 16, 4, 128, -1),      # pairs of heads, one block of rows
    (50, 100, 16, 16, 128, -1),     # pairs of row blocks, the second one without rows
    (50, 64, 16, 16, 64, -1),       # the same in at most 64 rows: one tile per CTA
    (6, 300, 16, 16, 128, -1),      # 288 tiles, 192 pairs: one tile per CTA
    (3, 768, 16, 16, 128, -1),      # 288 tiles, 144 pairs: one wave of pairs
    (1, 3001, 16, 16, 64, 512),     # 384 tiles, few key tiles each
    (15, 385, 16, 16, 64, 40),      # 960 tiles, the first key tile out of some rows' window
    (4, 900, 12, 4, 64, -1),        # three heads per KV head, 384 tiles and
    (5, 900, 12, 4, 64, -1),        # 480
])
def test_forward_on_both_sides_of_each_line(B, T, H, G, D, win):
    ext = backend.require_extension()
    torch.manual_seed(0)
    q, k, v = (torch.randn(B, T, n, D, device="cuda").bfloat16() for n in (H, G, G))
    scale = 1.0 / math.sqrt(D)
    out, lse = ext.attn_fwd_only(q, k, v, scale, win, None)
    assert ext.device_status() == 0
    for b in sorted({0, B // 2, B - 1}):
        ref, lse_ref = attention_ref(q[b:b + 1], k[b:b + 1], v[b:b + 1], scale, (win, 0) if win >= 0 else (-1, -1), None, None, True)
        # P and the result are rounded to bf16 (2^-9 each, the errors of P average out)
        assert float((out[b:b + 1].float() - ref).norm() / ref.norm()) < 2.0 ** -7
        assert float((lse[b:b + 1] - lse_ref).abs().max()) < 1e-3
