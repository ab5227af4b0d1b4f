"""Fixed-length document offsets against the compact list they stand for."""
import pytest
import torch

from archscale_b200.models.gated_deltanet import seq_idx_from_cu_seqlens
from archscale_b200.models.gpt import document_offsets
from archscale_b200.ops.attention import _build_mask, doc_end_from_cu_seqlens, row_start_from_cu_seqlens
from archscale_b200.ops.selective_scan import _reset_flags, selective_scan, selective_scan_ref


@pytest.mark.parametrize("eos", [[], [0], [9], [4], [0, 1, 2], [3, 9], list(range(10)), [0, 8, 9]])
def test_document_offsets(eos):
    T = 10
    is_eos = torch.zeros(T, dtype=torch.bool)
    is_eos[eos] = True
    compact = torch.tensor([0] + [e + 1 for e in eos if e + 1 < T] + [T], dtype=torch.int32)
    cu = document_offsets(is_eos)
    assert cu.dtype == torch.int32 and cu.numel() == T + 1
    assert torch.equal(cu[:compact.numel()], compact) and bool((cu[compact.numel():] == T).all())
    for f in (row_start_from_cu_seqlens, doc_end_from_cu_seqlens, _reset_flags, seq_idx_from_cu_seqlens):
        assert torch.equal(f(cu, T), f(compact, T)), f.__name__
    assert torch.equal(_build_mask(T, T, "cpu", (3, 0), cu), _build_mask(T, T, "cpu", (3, 0), compact))
    torch.manual_seed(0)
    u, d, B, C = torch.randn(1, 4, T), torch.rand(1, 4, T), torch.randn(1, 16, T), torch.randn(1, 16, T)
    A, D = -torch.rand(4, 16), torch.randn(4)
    y = selective_scan(u, d, A, B, C, D, cu_seqlens=cu)
    assert torch.allclose(y, selective_scan_ref(u, d, A, B, C, D, cu_seqlens=compact), atol=1e-5)
