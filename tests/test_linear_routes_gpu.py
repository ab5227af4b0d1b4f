"""Fused linear routes on the GPU: what they must not lose of the layers they stand for."""
import pytest
import torch
import torch.nn.functional as F

from archscale_b200.config import Config
from archscale_b200.models.gpt import LLaMAMLP
from archscale_b200.models.layers import Linear
from archscale_b200.ops import backend, gemm, swiglu_packed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("neighbours", [False, True])
@pytest.mark.parametrize("T", [8, 41, 64, 65, 72])
def test_hooks_of_the_projections_act_at_every_token_count(T, neighbours):
    torch.manual_seed(0)
    layers = [Linear(256, n, bias=False, device="cuda", dtype=torch.bfloat16) for n in (256, 64, 64)]
    if neighbours:
        flat = torch.cat([l.weight.detach() for l in layers])
        for l, w in zip(layers, flat.split([256, 64, 64])):
            l.weight = torch.nn.Parameter(w)
    x = torch.randn(1, T, 256, device="cuda").bfloat16()
    for grad in (False, True):
        with torch.set_grad_enabled(grad):
            plain = list(gemm.linear_multi(x, layers))
            h = layers[0].register_forward_hook(lambda m, a, y: y + 1)
            layers[2].forward = lambda x: x.new_zeros(*x.shape[:-1], 64)
            y = gemm.linear_multi(x, layers, keep_fused=True)
            assert not torch.is_tensor(y)
            tol = dict(rtol=2.0 ** -7, atol=2.0 ** -7)        # the fused product may sum in another order: one rounding to bf16 each
            torch.testing.assert_close(y[0], plain[0] + 1, **tol)
            torch.testing.assert_close(y[1], plain[1], **tol)
            assert not y[2].any()
            h.remove()
            del layers[2].forward


@pytest.mark.parametrize("T", [41, 64, 65, 72])
def test_a_hook_on_the_up_projection_acts_at_every_token_count(T):
    cfg = Config.from_name("transformer_gqa4_d8", intermediate_size=704)
    mlp = LLaMAMLP(cfg).cuda().bfloat16()
    mlp.reset_parameters()
    mlp.w1.register_forward_hook(lambda m, a, y: torch.zeros_like(y))
    with torch.no_grad():
        y, _ = mlp(torch.randn(1, T, cfg.n_embd, device="cuda").bfloat16(), 0)
    assert not y.any()


@pytest.mark.parametrize("T", [65, 257, 1001, 4099])
def test_odd_token_counts_without_gradients_run_the_library(T):
    torch.manual_seed(0)
    x, w = torch.randn(T, 256, device="cuda").bfloat16(), (torch.randn(264, 256, device="cuda") / 16).bfloat16()
    n0 = backend.launches()
    with torch.no_grad():
        y = gemm.linear(x, w)
    assert backend.launches() == n0 and torch.equal(y, F.linear(x, w))
    gemm.linear(x, w.requires_grad_())                       # with gradients: the own GEMM, whose backward pays
    assert backend.launches() == n0 + 1
    with torch.no_grad():
        gemm.linear(x[:T // 8 * 8], w)
        assert backend.launches() == n0 + 2


@pytest.mark.parametrize("one_cta", [False, True])
@pytest.mark.parametrize("T,N,off", [(1, 512, 0), (8, 512, 0), (64, 520, 0), (67, 512, 4), (1000, 512, 8), (1001, 264, 0), (1024, 512, 0)])
def test_a_bias_is_rounded_once_on_the_own_kernel(T, N, off, one_cta):
    """`off`: elements between a 32-byte boundary and the bias (no 16-byte boundary: copied; no 32-byte one: the narrow epilogue)."""
    torch.manual_seed(3)
    x, w = (torch.randn(T, 256, device="cuda") * 0.5).bfloat16(), (torch.randn(N, 256, device="cuda") * 0.5).bfloat16()
    b = (torch.randn(N + 16, device="cuda") * 2.0 ** -8).bfloat16()[off:off + N].requires_grad_()
    ext = backend.require_extension()
    was = ext.set_gemm_pair(not one_cta)
    try:
        n0 = backend.launches()
        y = gemm.linear(x, w, b)
        assert backend.launches() == n0 + 1
    finally:
        ext.set_gemm_pair(was)
    ref = x.double() @ w.double().t() + b.double()
    # half an ulp (at most 2^-8 of the value), and fp32 sums of 256 products of magnitude below 8
    assert bool(((y.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 256 * 8 * 2.0 ** -24).all())
    # two roundings leave errors of up to a whole ulp: with one, no element is further off than the library's by more than the sums' error
    lib = F.linear(x, w, b)
    assert bool(((y.double() - ref).abs() <= (lib.double() - ref).abs() + 2 * 256 * 8 * 2.0 ** -24).all())
    db, = torch.autograd.grad(y, b, torch.ones_like(y))
    assert torch.equal(db, torch.full_like(db, T))


@pytest.mark.parametrize("T", [41, 67, 72])
def test_transforms_and_traces_of_linear_layers(T):
    torch.manual_seed(5)
    x, w = (torch.randn(T, 128, device="cuda") / 8).bfloat16(), (torch.randn(64, 128, device="cuda") / 8).bfloat16()
    want = F.linear(x, w)
    for grad in (False, True):
        with torch.set_grad_enabled(grad):
            torch.testing.assert_close(torch.vmap(lambda r: gemm.linear(r, w))(x[:, None])[:, 0], want, rtol=2.0 ** -7, atol=2.0 ** -9)
            y, t = torch.func.jvp(lambda x: gemm.linear(x, w), (x,), (x,))
            torch.testing.assert_close(t, want, rtol=2.0 ** -7, atol=2.0 ** -9)
    assert not torch.jit.trace(lambda x: gemm.linear(x, w), x, check_trace=False).graph.findNode("prim::PythonOp")


def _penalty(fn, x, ws):
    """Gradients of the squared norm of an input gradient, as a gradient penalty takes them."""
    x = x.clone().requires_grad_()
    ws = [w.clone().requires_grad_() for w in ws]
    gx, = torch.autograd.grad(fn(x, ws).float().square().sum(), x, create_graph=True)
    return torch.autograd.grad(gx.float().square().sum(), [x, *ws])


@pytest.mark.parametrize("T", [41, 67, 72])
def test_second_derivatives_of_linear_layers(T):
    torch.manual_seed(4)
    x = (torch.randn(T, 128, device="cuda") / 8).bfloat16()
    flat = (torch.randn(96, 128, device="cuda") / 8).bfloat16()
    b = torch.zeros(64, device="cuda", dtype=torch.bfloat16)

    def multi(x, ws):
        layers = [Linear(128, n, bias=False, device="cuda", dtype=torch.bfloat16) for n in (64, 32)]
        for l, w in zip(layers, ws[0].split([64, 32])):
            del l.weight
            l.weight = w                                       # neighbours in one buffer, with a graph behind them
        return torch.cat(gemm.linear_multi(x, layers), -1)

    lib = lambda x, ws: F.linear(x, ws[0])
    for fn, ref, ws in ((lambda x, ws: gemm.linear(x, ws[0], b), lib, [flat[:64]]), (lambda x, ws: gemm.linear(x, ws[0]), lib, [flat[:64]]),
                        (multi, lib, [flat])):
        for got, want in zip(_penalty(fn, x, ws), _penalty(ref, x.float(), [w.float() for w in ws])):
            # four products in a row, a rounding to bf16 (2^-9) after each, none amplified
            assert float((got.float() - want).norm() / want.norm()) < 2.0 ** -6


@pytest.mark.parametrize("T", [67, 72])
def test_an_input_off_the_16_byte_grid_is_taken(T):
    x = torch.randn(T * 256 + 4, device="cuda").bfloat16()[4:].view(T, 256)
    w = (torch.randn(128, 256, device="cuda") / 16).bfloat16()
    y = gemm.linear_swiglu(x, w)
    y = y if y is not None else swiglu_packed(gemm.linear(x, w))
    g, u = (x.double() @ w.double().t()).chunk(2, -1)
    assert float((y.double() - F.silu(g) * u).norm() / (F.silu(g) * u).norm()) < 2.0 ** -7     # three roundings to bf16


def test_the_one_cta_switch_steers_products_of_few_rows(monkeypatch):
    x, w = torch.randn(16, 64, device="cuda").bfloat16(), torch.randn(64, 64, device="cuda").bfloat16()
    with torch.no_grad():
        assert gemm._skinny_ok(x, (w,))
        monkeypatch.setenv("ARCHSCALE_B200_GEMM", "1cta")
        gemm._one_cta.cache_clear()
        assert not gemm._skinny_ok(x, (w,))
    monkeypatch.undo()
    gemm._one_cta.cache_clear()


@pytest.mark.parametrize("one_cta", [False, True])
@pytest.mark.parametrize("T", [65, 257, 4099])
def test_odd_token_counts_run_one_own_launch_per_product(T, one_cta):
    torch.manual_seed(6)
    x, w, dy = ((torch.randn(*s, device="cuda") * 0.5).bfloat16() for s in ((T, 136), (264, 136), (T, 264)))
    ext, acc = backend.require_extension(), torch.full((264, 136), 0.25, device="cuda")
    ref = dy.double().t() @ x.double()
    was = ext.set_gemm_pair(not one_cta)
    try:
        for fn, want, tol in ((lambda: gemm.matmul_nt(x, w), x.double() @ w.double().t(), 2.0 ** -8),
                              (lambda: gemm.matmul_nn(dy, w), dy.double() @ w.double(), 2.0 ** -8),
                              (lambda: gemm.matmul_tn(dy, x), ref, 2.0 ** -8),
                              (lambda: gemm.matmul_tn_acc_(acc, dy, x), ref + 0.25, 1e-5)):        # fp32 sums of bf16 products
            n0 = backend.launches()
            got = fn()
            assert backend.launches() == n0 + 1
            assert float((got.double() - want).norm() / want.norm()) < tol
    finally:
        ext.set_gemm_pair(was)
    assert ext.device_status() == 0


def test_the_gathering_gemm_adds_the_bias():
    """Both ranks' shards on one device, as the launch pulls them; the copying CTAs and the product are one kernel."""
    torch.manual_seed(7)
    ext, (M, N, K) = backend.require_extension(), (264, 512, 256)
    shards = [(0.05 * torch.randn(N * K // 2, device="cuda")).bfloat16() for _ in range(2)]
    a, b = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(N, device="cuda").bfloat16()
    dst = torch.zeros(N * K, device="cuda", dtype=torch.bfloat16)
    flags = torch.zeros((dst.numel() * 2 + 256 * 1024 - 1) // (256 * 1024), dtype=torch.int32, device="cuda")
    args = (a, [t.data_ptr() for t in shards], 0, dst, N * K, 0, N, flags)
    y = ext.ag_gemm(*args, 1, 0, 16, gemm.bias_row(b))
    ref = a.double() @ torch.cat(shards).view(N, K).double().t()
    assert float((y.double() - ref - b.double()).norm() / ref.norm()) < 2.0 ** -8          # one rounding to bf16
    assert float((ext.ag_gemm(*args, 2, 0, 16).double() - ref).norm() / ref.norm()) < 2.0 ** -8
    assert ext.device_status() == 0
