"""Which layers and weights the fused linear routes may take."""
import torch

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
