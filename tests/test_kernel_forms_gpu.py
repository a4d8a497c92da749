"""Kernels that serve some sizes in a form of their own, against the form for any size or float64."""
from types import SimpleNamespace

import pytest
import torch

from fastllm_py_b200.native import ops

pytestmark = pytest.mark.gpu


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("dim", [4, 100, 1024, 1028, 2048, 4100, 8192, 12288])
def test_norm_add_norm_in_wide_and_single_accesses(dim):
    """Buffers that 16-byte loads can read and ones that they cannot give the same bits."""
    torch.manual_seed(dim)
    y, x = torch.randn(3, dim, device="cuda").to(torch.bfloat16), torch.randn(3, dim, device="cuda")
    wa, wb = (1 + 0.2 * torch.randn(2, dim, device="cuda")).to(torch.bfloat16)
    outs = []
    for shift in (0, 1):
        xs = torch.empty(3 * dim + 4, device="cuda")[shift:shift + 3 * dim].view(3, dim)
        xs.copy_(x)
        out = torch.empty(3, dim, device="cuda", dtype=torch.bfloat16)
        ops.sandwich_norm(xs, y, wa, 1e-5, wb, 1e-6, out)
        outs.append((xs.clone(), out))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
    yd = y.double()
    ref = x.double() + yd / torch.sqrt((yd * yd).mean(-1, keepdim=True) + 1e-5) * wa.double()
    assert float((outs[0][0].double() - ref).abs().max()) <= 1e-5 * float(ref.abs().max())   # (sums of 32 bits)
