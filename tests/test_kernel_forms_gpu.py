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


@pytest.mark.parametrize("dim, vdim", [(128, 128), (128, 40), (64, 64), (20, 7), (256, 96)])
@pytest.mark.parametrize("lens", [[1, 2], [3], [17, 18, 19], [36, 0, 5], [150]])
def test_delta_scan_that_looks_ahead(lens, dim, vdim):
    """Against the recurrence in float64, and no further from it than twice the other kernel (both sum the same products in
    32 bits, in another order); states carried over and fresh ones."""
    torch.manual_seed(dim + sum(lens))
    heads, kv_heads, n = 4, 2, sum(lens)
    qk, hv = kv_heads * dim, heads * vdim
    q, k = torch.randn(n, kv_heads, dim, device="cuda"), torch.randn(n, kv_heads, dim, device="cuda")
    k /= k.norm(dim=-1, keepdim=True)
    q *= dim ** -0.5 / q.norm(dim=-1, keepdim=True)
    v = torch.randn(n, heads, vdim, device="cuda")
    beta, decay = torch.rand(n, heads, device="cuda"), 1.0 - 0.1 * torch.rand(n, heads, device="cuda")
    rows = torch.cat([q.flatten(1), k.flatten(1), v.flatten(1), beta, decay, torch.zeros(n, hv, device="cuda")], 1).contiguous()
    state0 = torch.randn(len(lens), hv * dim, device="cuda")
    starts = [sum(lens[:r]) for r in range(len(lens) + 1)]
    ctx = [5 * (r % 2) for r in range(len(lens))]
    step = SimpleNamespace(req_start=i32(starts), req_ctx=i32(ctx), req_qlen=i32(lens), req_slot=i32(list(range(len(lens)))),
                           n_requests=len(lens))
    of = torch.arange(heads, device="cuda") // (heads // kv_heads)
    want, want_state = torch.zeros(n, heads, vdim, dtype=torch.float64, device="cuda"), state0.double().clone()
    for r, m in enumerate(lens):
        S = state0[r].double().view(heads, vdim, dim) * (ctx[r] > 0)
        for t in range(starts[r], starts[r] + m):
            kt, qt = k[t, of].double()[:, :, None], q[t, of].double()[:, :, None]
            S = S * decay[t].double()[:, None, None]
            u = beta[t].double()[:, None, None] * (v[t].double()[:, :, None] - S @ kt)
            S = S + u @ kt.transpose(1, 2)
            want[t] = (S @ qt)[:, :, 0]
        want_state[r] = S.flatten()
    errors = []
    for ahead in (False, True):
        work, state = rows.clone(), state0.clone()
        ops.delta_scan(work, state, step, heads, kv_heads, dim, vdim, ahead=ahead)
        got = work[:, 2 * qk + hv + 2 * heads:].view(n, heads, vdim)
        errors.append((float((got.double() - want).abs().max()), float((state.double() - want_state).abs().max())))
    assert errors[1][0] <= 2 * errors[0][0] + 1e-6 and errors[1][1] <= 2 * errors[0][1] + 1e-6, errors
    assert errors[1][0] < 1e-4 * max(1.0, float(want.abs().max()))
