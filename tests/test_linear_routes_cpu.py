"""Which layers and weights the fused linear routes may take."""
import torch
import torch.nn.utils.parametrize

from archscale_b200.models.layers import Linear
from archscale_b200.ops import gemm


def test_neighbours_in_memory_are_adjacent_only_inside_one_storage():
    flat = torch.arange(24.0).view(6, 4)
    assert gemm._adjacent([flat[:2], flat[2:3], flat[3:]])
    assert torch.equal(gemm._cat_view([flat[:2], flat[2:3], flat[3:]]), flat)
    assert not gemm._adjacent([flat[:2], flat[3:]])
    raw = bytearray(96)                                  # two storages over neighbouring memory, as an allocator may place them
    a = torch.frombuffer(raw, dtype=torch.float32, count=8, offset=0).view(2, 4)
    b = torch.frombuffer(raw, dtype=torch.float32, count=16, offset=32).view(4, 4)
    assert a.data_ptr() + 32 == b.data_ptr()
    assert not gemm._adjacent([a, b])


def test_only_a_layer_that_is_a_product_and_nothing_else_may_be_passed_by():
    layer = lambda **kw: Linear(8, 8, **{"bias": False, **kw})
    assert gemm.plain_linear(layer())
    assert not gemm.plain_linear(layer(bias=True)) and not gemm.plain_linear(torch.nn.Linear(8, 8, bias=False))
    for register in ("register_forward_hook", "register_forward_pre_hook", "register_full_backward_hook", "register_full_backward_pre_hook"):
        l = layer()
        h = getattr(l, register)(lambda *a: None)
        assert not gemm.plain_linear(l), register
        h.remove()
        assert gemm.plain_linear(l)
    h = torch.nn.modules.module.register_module_forward_hook(lambda *a: None)
    assert not gemm.plain_linear(layer())
    h.remove()
    l = layer()
    l.forward = lambda x: x
    assert not gemm.plain_linear(l)
    l = layer()
    l.mxfp8 = True
    assert not gemm.plain_linear(l)
    plain = Linear.forward
    try:
        Linear.forward = lambda self, x: x
        assert not gemm.plain_linear(layer())
    finally:
        Linear.forward = plain
    l = layer()
    torch.nn.utils.parametrize.register_parametrization(l, "weight", torch.nn.Identity())
    assert not gemm.plain_linear(l)
