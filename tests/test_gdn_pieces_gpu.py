"""64×64 pieces of the gated delta rule: the kernels against the element-wise formulas in fp64, forward and backward."""
import pytest
import torch

from archscale_b200.ops.gated_delta_rule import _ColsFn, _MaskFn

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30))


@pytest.mark.parametrize("shape,decay", [((1, 1), 0.05), ((3, 43), 0.5), ((2, 5), 8.0)])     # weak, ordinary, vanishing after a few tokens
def test_pieces_match_formulas(shape, decay):
    torch.manual_seed(0)
    dev = "cuda"
    Gk, Gq = (torch.randn(*shape, 64, 64, device=dev).requires_grad_() for _ in range(2))
    gc = torch.cumsum(-torch.rand(*shape, 64, device=dev) * decay, -1).requires_grad_()
    beta = (torch.rand(*shape, 64, device=dev) * 2).requires_grad_()
    T = torch.randn(*shape, 64, 64, device=dev).requires_grad_()
    outs = _MaskFn.apply(Gk, Gq, gc, beta) + _ColsFn.apply(T, gc, beta)
    gs = [torch.randn_like(o) for o in outs]
    leaves = [Gk, Gq, gc, beta, T]
    got = torch.autograd.grad(outs, leaves, gs)

    r = [t.detach().double().requires_grad_() for t in leaves]
    low = torch.ones(64, 64, device=dev, dtype=torch.bool).tril()
    dec = torch.exp((r[2].unsqueeze(-1) - r[2].unsqueeze(-2)).masked_fill(~low, 0.0))
    ref = ((r[0] * dec * r[3].unsqueeze(-1)).masked_fill(~low.tril(-1), 0.0), (r[1] * dec).masked_fill(~low, 0.0),
           r[4] * r[3].unsqueeze(-2), r[4] * (r[3] * torch.exp(r[2])).unsqueeze(-2))
    want = torch.autograd.grad(ref, r, [g.double() for g in gs])
    for o, w in zip(outs, ref):
        assert _rel(o, w) < (1e-6 if o.dtype == torch.float32 else 2.0 ** -8)
    # Gram gradients are rounded to bf16; the other gradients are fp32 (sums of up to 192 products)
    for name, a, b in zip(("Gk", "Gq", "gc", "beta", "T"), got, want):
        assert _rel(a, b) < (2.0 ** -8 if name in ("Gk", "Gq") else 5e-6), name
    again = torch.autograd.grad(_MaskFn.apply(Gk, Gq, gc, beta) + _ColsFn.apply(T, gc, beta), leaves, gs)
    assert all(torch.equal(a, b) for a, b in zip(got, again))
