"""Selective scan on the branches its kernels choose by size, alignment and type."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _scan_case(B, L, Di, dtype, packed, gate, shift):
    """Operands as slices of wider rows; ``shift`` elements of offset decide whether vector loads are possible."""
    torch.manual_seed(5)
    dev = "cuda"
    wide = lambda n: torch.randn(B, L, n + 8, device=dev).to(dtype)[..., shift:shift + n].detach().requires_grad_(True)
    u, z = wide(Di), (wide(Di) if gate else None)
    delta = (torch.randn(B, L, Di + 8, device=dev) * 0.5).to(dtype)[..., shift:shift + Di].detach().requires_grad_(True)
    Bm, Cm = wide(16), wide(16)
    A = (-torch.exp(torch.rand(Di, 16, device=dev) * 2 - 1)).requires_grad_(True)
    D, bias = torch.randn(Di, device=dev).requires_grad_(True), (torch.randn(Di, device=dev) * 0.3).requires_grad_(True)
    cu = torch.tensor([0, 1, 31, 32, 33, 64, L], device=dev, dtype=torch.int32) if packed else None
    return u, delta, A, Bm, Cm, D, bias, z, cu


@pytest.mark.parametrize("B,L,Di,dtype,packed,gate,shift", [
    (4, 97, 3072, torch.float32, False, True, 0),       # B·Di = 12288: four states per thread, one step into the fourth 32-step tile
    (4, 33, 3088, torch.bfloat16, False, False, 0),
    (4, 40, 3072, torch.float32, False, True, 1),       # rows that start at odd elements: scalar loads
    (2, 65, 48, torch.bfloat16, False, True, 3),        # two states per thread
    (1, 129, 12288, torch.float32, True, True, 0),      # four states per thread with documents, breaks on and beside tile edges
    (1, 100, 64, torch.float32, True, False, 2),
    (1, 1, 16, torch.float32, False, True, 0),
    (1, 1536, 48, torch.float32, False, True, 0),       # time in three parts
    (1, 1601, 32, torch.float32, True, True, 0),        # parts of 576 steps, the last one shorter; breaks in the first part only
    (2, 2049, 32, torch.bfloat16, False, False, 1),     # one step into the last 64-step tile
])
def test_selective_scan_branches(B, L, Di, dtype, packed, gate, shift):
    from archscale_b200.ops.selective_scan import selective_scan, selective_scan_ref
    if packed and L < 65:
        pytest.skip("breaks up to 64")
    u, delta, A, Bm, Cm, D, bias, z, cu = _scan_case(B, L, Di, dtype, packed, gate, shift)
    y = selective_scan(u, delta, A, Bm, Cm, D, z=z, delta_bias=bias, delta_softplus=True, cu_seqlens=cu, channel_last=True)
    g = torch.randn(y.shape, device="cuda").to(dtype)
    leaves = [t for t in (u, delta, A, Bm, Cm, D, bias, z) if t is not None]
    grads = torch.autograd.grad(y, leaves, g)
    refs = [t.detach().float().clone().requires_grad_(True) for t in leaves]
    t = lambda v: v.transpose(1, 2)
    yr = t(selective_scan_ref(t(refs[0]), t(refs[1]), refs[2], t(refs[3]), t(refs[4]), refs[5], z=t(refs[7]) if gate else None,
                              delta_bias=refs[6], delta_softplus=True, cu_seqlens=cu))
    gr = torch.autograd.grad(yr, refs, g.float())
    # fp32: sums of a few hundred products (2^-24 each) against another order; bf16: one rounding (2^-9) of every stored result
    tol = 2e-5 if dtype == torch.float32 else 8e-3
    for a, r in zip((y, *grads), (yr, *gr)):
        assert float((a.float() - r).norm()) <= tol * float(r.norm()) + 1e-6
