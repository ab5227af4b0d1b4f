"""Mamba projections whose feature counts are no multiple of 8: the module is called, and the widened product is the product."""
import pytest
import torch

from archscale_b200.models.mamba import Mamba


@pytest.mark.parametrize("d_model", [64, 128, 1984])
def test_projections_are_called(d_model):
    m = Mamba(d_model, expand=1 if d_model > 1000 else 2)
    m.reset_parameters()
    seen = []
    for name in ("in_proj", "x_proj", "out_proj"):
        getattr(m, name).register_forward_hook(lambda mod, args, out, name=name: seen.append((name, tuple(out.shape))))
    m(torch.randn(2, 3, d_model))
    assert seen == [("in_proj", (2, 3, 2 * m.d_inner)), ("x_proj", (2, 3, m.dt_rank + 32)), ("out_proj", (2, 3, d_model))]


@pytest.mark.gpu
@pytest.mark.parametrize("B,L", [(1, 2040), (1, 2048), (1, 2049), (2, 2100)])
@pytest.mark.parametrize("d_model", [1088, 1024])
def test_mixer_on_widened_projections(d_model, B, L):
    """dt_rank 68 (x_proj 100 features, dt_proj 68 inputs) and, beside it, 64; output and gradients against the same mixer in fp32."""
    dev = "cuda"
    m = Mamba(d_model).to(dev)
    m.reset_parameters()
    ref = Mamba(d_model).to(dev)
    with torch.no_grad():
        for p in m.parameters():
            p.copy_(p.bfloat16().float())
    ref.load_state_dict(m.state_dict())
    m = m.bfloat16()
    for n in ("A_log", "D"):
        getattr(m, n).data = getattr(ref, n).data.clone()
    seen = []
    m.x_proj.register_forward_hook(lambda mod, args, out: seen.append(tuple(out.shape)))
    x = torch.randn(B, L, d_model, device=dev).bfloat16()
    g = torch.randn(B, L, d_model, device=dev).bfloat16()
    xs, xr = x.clone().requires_grad_(True), x.float().requires_grad_(True)
    y, yr = m(xs)[0], ref(xr)[0]
    assert seen == [(B, L, m.dt_rank + 32)] and y.shape == yr.shape
    y.backward(g)
    yr.backward(g.float())
    # six bf16 roundings (2^-9 each) between input and output, twice that through the backward
    close = lambda a, r, tol: float((a.float() - r).norm()) <= tol * float(r.norm())
    assert close(y, yr, 1e-2) and close(xs.grad, xr.grad, 2e-2)
    for (n, p), (_, r) in zip(m.named_parameters(), ref.named_parameters()):
        assert p.grad.shape == p.shape and close(p.grad, r.grad, 2e-2), n


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [2048, 2049, 8193])
@pytest.mark.parametrize("k,n", [(3968, 156), (124, 3968), (68, 100), (100, 68)])
def test_widened_product(rows, k, n):
    """Output and both gradients against fp64, and no further off than the library's product on the unpadded operands."""
    from archscale_b200.ops import gemm
    dev = "cuda"
    x = torch.randn(rows, k, device=dev).bfloat16().requires_grad_(True)
    w = (torch.randn(n, k, device=dev) / k ** 0.5).bfloat16().requires_grad_(True)
    g = torch.randn(rows, n, device=dev).bfloat16()
    assert gemm.widened_ok(x, w)
    y = gemm.linear_widened(x, w)
    lib = torch.nn.functional.linear(x, w)
    assert y.shape == lib.shape
    xd, wd = x.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
    yd = xd @ wd.t()
    for a, b, r in zip((y, *torch.autograd.grad(y, (x, w), g)), (lib, *torch.autograd.grad(lib, (x, w), g)),
                       (yd, *torch.autograd.grad(yd, (xd, wd), g.double()))):
        err = lambda t: float((t.double() - r).norm() / r.norm())
        assert a.shape == r.shape and err(a) <= 2 ** -9 and err(a) <= 1.05 * err(b) + 1e-5
