"""Segment update with an fp32 direction (embeddings and heads under the hyperball rule) against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 4092, 4096, 4100, 1_000_004])
@pytest.mark.parametrize("u_dtype", [torch.float32, torch.bfloat16])
def test_seg_update(n, u_dtype):
    from archscale_b200.ops import backend
    ext = backend.require_extension()
    torch.manual_seed(12)
    x = torch.randn(n, device="cuda")
    u = torch.randn(n, device="cuda").to(u_dtype)
    x0 = x.double().clone()
    bounds, kidx = torch.tensor([0, n], device="cuda"), torch.tensor([2], dtype=torch.int32, device="cuda")
    coef, acc = torch.tensor([9.0, 9.0, 0.03, 9.0], device="cuda"), torch.zeros(4, device="cuda")
    ext.seg_update_(1, x, u, bounds, kidx, coef, acc)
    ref = x0 - coef[2].double() * u.double()
    assert float((x.double() - ref).abs().max()) <= 2 ** -23 * float(ref.abs().max())           # one fused multiply-add each
    sq = float(ref.square().sum())
    assert abs(float(acc[2]) - sq) <= 1e-5 * sq and float(acc[[0, 1, 3]].abs().max()) == 0.0    # fp32 sum of n squares
    before = x.clone()
    ext.seg_update_(2, x, None, bounds, kidx, coef, None)
    assert torch.equal(x, before * coef[2])
