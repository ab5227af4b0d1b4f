"""QK-norm + rotary kernels (half a warp per head) at head counts and token counts that leave half a step over."""
import pytest
import torch

from archscale_b200.ops import backend
from archscale_b200.ops.rope import qk_norm_rope_ref, qkv_norm_rope, qkv_norm_rope_supported

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,H,G,D,norm,rot,grouped", [
    (1, 13, 3, 1, 128, True, True, False), (2, 7, 5, 5, 64, True, True, False), (1, 1, 7, 1, 128, True, False, False),
    (1, 700, 6, 3, 64, False, True, False), (3, 129, 16, 4, 128, True, True, False),
    (1, 13, 6, 2, 128, True, True, True), (2, 7, 5, 5, 64, True, True, True), (1, 1, 14, 2, 128, True, False, True),
    (1, 700, 6, 3, 64, False, True, True), (3, 129, 16, 4, 128, True, True, True)])
def test_qkv_norm_rope_matches_reference(B, T, H, G, D, norm, rot, grouped):
    torch.manual_seed(0)
    dev = "cuda"
    x = torch.randn(B, T, (H + 2 * G) * D, device=dev).bfloat16()
    w = [(torch.rand(D, device=dev) + 0.5).requires_grad_() for _ in range(2)] if norm else [None, None]
    ang = torch.rand(T, D // 2, device=dev) * 6
    cs = [ang.cos().bfloat16(), ang.sin().bfloat16()] if rot else [None, None]
    leaf = x.clone().requires_grad_()
    assert qkv_norm_rope_supported(leaf, H, G, cs[0], w[0])
    n0 = backend.launches()
    outs = qkv_norm_rope(leaf, H, G, grouped, w[0], w[1], cs[0], cs[1], 1e-5)
    assert backend.launches() > n0
    gs = [torch.randn_like(o) for o in outs]
    grads = torch.autograd.grad(outs, [leaf] + [t for t in w if norm], gs)

    ref_leaf = x.float().requires_grad_()
    ref_w = [t.detach().clone().requires_grad_() if norm else None for t in w]
    if grouped:
        y = ref_leaf.view(B, T, G, H // G + 2, D)
        q, k, v = y[..., :-2, :].reshape(B, T, H, D), y[..., -2, :], y[..., -1, :]
    else:
        y = ref_leaf.view(B, T, H + 2 * G, D)
        q, k, v = y[:, :, :H], y[:, :, H:H + G], y[:, :, H + G:]
    cf = [c.float() if c is not None else None for c in cs]
    qr, kr = qk_norm_rope_ref(q, k, ref_w[0], ref_w[1], cf[0], cf[1], 1e-5)
    ref = torch.autograd.grad((qr, kr, v), [ref_leaf] + [t for t in ref_w if norm], [g.float() for g in gs])
    rel = lambda a, b: float((a.float() - b.float()).norm() / b.float().norm())
    # outputs and the projection's gradient are rounded once to bf16 (2^-9 relative); gain gradients are fp32 sums
    for a, b in zip(outs, (qr, kr, v)):
        assert rel(a, b) < 2.0 ** -8
    assert rel(grads[0], ref[0]) < 2.0 ** -8
    for a, b in zip(grads[1:], ref[1:]):
        assert rel(a, b) < 1e-4


@pytest.mark.parametrize("H,D", [(3, 128), (5, 64)])
def test_an_infinite_gradient_in_the_last_head_stays_infinite(H, D):
    """The steps over heads go past the last one where four do not divide their number: that adds nothing, not 0 · inf."""
    torch.manual_seed(1)
    x = torch.randn(1, 6, (H + 2) * D, device="cuda").bfloat16().requires_grad_()
    w = [(torch.rand(D, device="cuda") + 0.5).requires_grad_() for _ in range(2)]
    ang = torch.rand(6, D // 2, device="cuda") + 0.2
    q, k, v = qkv_norm_rope(x, H, 1, False, w[0], w[1], ang.cos().bfloat16(), ang.sin().bfloat16(), 1e-5)
    g = torch.randn_like(q)
    g[0, 4, H - 1, 5] = float("inf")
    dw, = torch.autograd.grad(q, w[0], g)
    assert not dw.isnan().any() and dw.isinf().nonzero().flatten().tolist() == [5, 5 + D // 2]
