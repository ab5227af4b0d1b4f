"""Decay factors of the delta rule's 64×64 blocks, element by element: e^x over all that a log-decay can be."""
import pytest
import torch

from archscale_b200.ops import backend

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo,hi", [(-1.0, 0.0), (-20.0, 0.0), (-110.0, -80.0), (80.0, 88.72)])
def test_decay_factors_are_accurate_everywhere(lo, hi):
    ext = backend.require_extension()
    n = 32
    gc = torch.linspace(lo, hi, n * 63, device="cuda").view(n, 63)
    gc = torch.cat([torch.zeros(n, 1, device="cuda"), gc], 1).contiguous()          # column 0: e^(gc_i − 0), no rounding in the difference
    one = torch.ones(n, 64, 64, device="cuda")
    beta = torch.ones(n, 64, device="cuda")
    A, _ = ext.gdn_mask_fwd(one, one, gc, beta)
    # what the formula gives element by element, bit for bit (the products are with one)
    assert torch.equal(A[:, 1:, 0], torch.exp(gc)[:, 1:])


def test_decay_factors_of_special_values():
    ext = backend.require_extension()
    gc = torch.zeros(1, 64, device="cuda")
    gc[0, 1:5] = torch.tensor([float("-inf"), -200.0, float("nan"), 200.0])
    one = torch.ones(1, 64, 64, device="cuda")
    A, qk = ext.gdn_mask_fwd(one, one, gc, torch.ones(1, 64, device="cuda"))
    col = A[0, 1:5, 0]
    assert col[0] == 0 and col[1] == 0 and bool(col[2].isnan()) and col[3] == float("inf")
    assert not A[0].triu().any() and not qk[0].triu(1).any()                         # what is masked stays zero beside them
