"""The kernels at the lengths and alignments where their splits can go wrong, each against a plain PyTorch
computation of the same operation."""
import pytest
import torch

import allreduce_proto_b200 as ar

pytestmark = pytest.mark.gpu


def values(n, dtype, seed, offset=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    if dtype in (torch.int32, torch.int64):
        t = torch.randint(-1000, 1000, (n + offset,), device="cuda", dtype=dtype, generator=g)
    else:
        t = (torch.rand(n + offset, device="cuda", generator=g) * 2 - 1).to(dtype)
    return t[offset:]


@pytest.mark.parametrize("offsets", [(0, 0), (1, 1), (3, 3), (1, 0), (4, 4)])
@pytest.mark.parametrize("types", [(torch.float32, torch.float32), (torch.float32, torch.bfloat16), (torch.bfloat16, torch.float32),
                                   (torch.float16, torch.float32), (torch.bfloat16, torch.bfloat16), (torch.float64, torch.float64),
                                   (torch.int64, torch.int64)])
def test_copy_scale_quanta_heads_and_tails(types, offsets):
    # One quantum per thread, 256 threads per block: lengths around a quantum, a block and several blocks; slices that
    # share an offset (peeled up to the boundary) and slices that do not (element by element).
    for n in (1, 3, 7, 8, 15, 16, 17, 33, 2047, 2048, 2049, 4096 + 5, 100003):
        x = values(n, types[0], n, offsets[0])
        guard = torch.full((n + offsets[1] + 8,), 7, device="cuda", dtype=types[1])
        y = guard[offsets[1]:offsets[1] + n]
        scale = 1.0 if types[0] == torch.int64 else 0.5
        ar.ops.copy_scale(x, y, scale=scale)
        assert torch.equal(y, (x.double() * scale).to(types[1])), n
        assert torch.all(guard[:offsets[1]] == 7) and torch.all(guard[offsets[1] + n:] == 7), n
