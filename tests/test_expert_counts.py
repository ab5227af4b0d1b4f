"""Tokens per expert without a host wait: values at the edges of the table, and memory that does not grow with tokens times experts."""
import pytest
import torch

from archscale_b200.ops.moe import COUNT_ROWS, expert_counts


@pytest.mark.parametrize("T", [0, 1, COUNT_ROWS - 1, COUNT_ROWS, COUNT_ROWS + 1, 3 * COUNT_ROWS + 5])
@pytest.mark.parametrize("E,K,dtype", [(1, 1, torch.int64), (64, 8, torch.int32)])
def test_counts_match_bincount(T, E, K, dtype):
    idx = torch.randint(0, E, (T, K), generator=torch.Generator().manual_seed(T)).to(dtype)
    for i in (idx, idx.t().contiguous().t()):
        assert torch.equal(expert_counts(i, E), torch.bincount(i.reshape(-1).long(), minlength=E).float())


@pytest.mark.gpu
def test_counts_need_a_bounded_table():
    T, E, K = 65536, 256, 4
    idx = torch.randint(0, E, (T, K), device="cuda", dtype=torch.int32)
    want = torch.bincount(idx.reshape(-1), minlength=E).float()
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    base = torch.cuda.memory_allocated()
    torch.cuda.set_sync_debug_mode("error")
    try:
        got = expert_counts(idx, E)
    finally:
        torch.cuda.set_sync_debug_mode("default")
    peak = torch.cuda.max_memory_allocated() - base
    assert torch.equal(got, want)
    assert peak <= T * K * 8 + COUNT_ROWS * E * 4 + (1 << 20)        # the 64-bit indices and the table (a row per token: 67 MB more)
