"""Kernels that serve some sizes in a form of their own, against the form for any size or float64."""
from types import SimpleNamespace

import pytest
import torch

from fastllm_py_b200.native import ops

pytestmark = pytest.mark.gpu


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("dim", [4, 100, 1024, 1028, 2048, 4100, 8192, 12256])
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


@pytest.mark.parametrize("size,heads,kv_heads,page", [(128, 4, 1, 16), (64, 6, 3, 8), (128, 2, 2, 128)])
@pytest.mark.parametrize("gate,sink", [(None, False), ("head", True), ("channel", False)])
def test_prompt_attention_over_rows_of_keys_and_values(size, heads, kv_heads, page, gate, sink):
    """tcgen05 tiles against the CUDA-core kernel (both round a row's result to bfloat16 once, tcgen05 the weights too: 2^-8 of
    the values' size each); what the last page holds behind a prompt's last token is not finite."""
    torch.manual_seed(size + heads)
    ctx, lens = [0, 130, 5, 1, 0], [300, 129, 1, 64, 2]
    per = [-(-(c + m) // page) for c, m in zip(ctx, lens)]
    cache = torch.randn(sum(per), kv_heads, page, 2 * size, device="cuda").to(torch.bfloat16)
    bt = torch.zeros(len(lens), max(per), dtype=torch.int32, device="cuda")
    for r, n in enumerate(per):
        bt[r, :n] = torch.arange(sum(per[:r]), sum(per[:r]) + n)
        rest = n * page - ctx[r] - lens[r]
        if rest:
            cache[int(bt[r, n - 1]), :, page - rest:, size:] = float("inf")
            cache[int(bt[r, n - 1]), :, page - rest:, :size] = float("nan")
    starts = [sum(lens[:r]) for r in range(len(lens) + 1)]
    n = starts[-1]
    step = SimpleNamespace(req_start=i32(starts), req_ctx=i32(ctx), req_qlen=i32(lens), n_requests=len(lens), q_lens=lens)
    tok_req = i32([r for r, m in enumerate(lens) for _ in range(m)])
    positions = i32([c + i for c, m in zip(ctx, lens) for i in range(m)])
    q = torch.randn(n, heads * size, device="cuda").to(torch.bfloat16)
    g = None if gate is None else torch.randn(n, heads if gate == "head" else heads * size, device="cuda").to(torch.bfloat16)
    s = torch.randn(heads, device="cuda") if sink else None
    want, got = torch.empty_like(q), torch.zeros_like(q)
    ops.sink_attention_simt(q, want, cache, bt, tok_req, positions, heads, kv_heads, size, size, None, 0, size ** -0.5, None, None,
                            None, s, page, gate=g)
    assert ops.sink_rows_takes(size, size, None, 0, None, None, None, page)
    ops.sink_attention_rows(q, got, cache, bt, step, heads, kv_heads, size, size ** -0.5, s, page, True, g)
    assert bool(got.isfinite().all())
    assert float((got.float() - want.float()).abs().max()) <= 2 ** -6 * float(want.float().abs().max())
    alone = torch.zeros_like(q)
    ops.sink_attention_rows(q, alone, cache, bt, step, heads, kv_heads, size, size ** -0.5, s, page, False, g)
    single = starts[2]
    assert not bool(alone[single].any()) and torch.equal(alone[:single], got[:single]) and torch.equal(alone[single + 1:], got[single + 1:])


def prompts_over_rows(lens, size, heads, kv_heads, page, seed):
    """Queries, a cache of rows k | v in shuffled pages and a step for requests of (cached, new) tokens."""
    torch.manual_seed(seed)
    per = [-(-(c + m) // page) for c, m in lens]
    cache = torch.randn(sum(per), kv_heads, page, 2 * size, device="cuda").to(torch.bfloat16)
    order = torch.randperm(sum(per), device="cuda").to(torch.int32)
    bt = torch.zeros(len(lens), max(per), dtype=torch.int32, device="cuda")
    for r, n in enumerate(per):
        bt[r, :n] = order[sum(per[:r]):sum(per[:r]) + n]
    starts = [sum(m for _, m in lens[:r]) for r in range(len(lens) + 1)]
    step = SimpleNamespace(req_start=i32(starts), req_ctx=i32([c for c, _ in lens]), req_qlen=i32([m for _, m in lens]),
                           n_requests=len(lens), q_lens=[m for _, m in lens], ctx_lens=[c for c, _ in lens])
    return torch.randn(starts[-1], heads * size, device="cuda").to(torch.bfloat16), cache, bt, step


@pytest.mark.parametrize("size,heads,kv_heads,page", [(128, 4, 2, 16), (64, 6, 3, 8), (128, 2, 1, 64), (64, 2, 2, 128)])
@pytest.mark.parametrize("sink,gate", [(None, None), (1.0, "head"), (60.0, "channel"), (-60.0, None)])
def test_both_prompt_kernels_over_rows_give_the_same_bits(size, heads, kv_heads, page, sink, gate):
    """Prompts of a few tokens and of many key blocks (the ring goes round; more than 64 blocks are asked for at once), at
    positions that are and are not multiples of 64, sinks far above and far below the scores; against float64 the
    weights' and the result's rounding to bfloat16, 2^-9 of the largest value each."""
    lens = [(0, 300), (4300, 150), (130, 129), (63, 66), (64, 128), (1, 1), (700, 1), (0, 2), (500, 17), (0, 2)]
    q, cache, bt, step = prompts_over_rows(lens, size, heads, kv_heads, page, size + heads)
    n, scale = q.shape[0], 3 * size ** -0.5
    g = None if gate is None else torch.randn(n, heads if gate == "head" else heads * size, device="cuda").to(torch.bfloat16)
    s = None if sink is None else torch.randn(heads, device="cuda") + sink
    want, got = torch.empty_like(q), torch.zeros_like(q)
    ops.sink_attention_mma(q, want, cache, bt, step, heads, kv_heads, size, size, None, 0, scale, None, None, None, s, page, gate=g)
    ops.sink_attention_rows(q, got, cache, bt, step, heads, kv_heads, size, scale, s, page, True, g)
    assert torch.equal(got, want)
    start = 0
    for r, (c, m) in enumerate(lens):
        kv = cache[bt[r, :-(-(c + m) // page)].long()].permute(1, 0, 2, 3).reshape(kv_heads, -1, 2 * size)[:, :c + m].double()
        kv = kv.repeat_interleave(heads // kv_heads, 0)
        scores = q[start:start + m].view(m, heads, size).transpose(0, 1).double() @ kv[..., :size].transpose(1, 2) * scale
        scores += torch.full((m, c + m), float("-inf"), device="cuda", dtype=torch.double).triu(c + 1)
        extra = torch.full((heads, m, 1), float("-inf"), device="cuda", dtype=torch.double) if s is None else s.double().view(-1, 1, 1).expand(-1, m, 1)
        ref = (torch.cat([scores, extra], -1).softmax(-1)[..., :-1] @ kv[..., size:]).transpose(0, 1).reshape(m, heads * size)
        if g is not None:
            gate_of = g[start:start + m].double().sigmoid()
            ref = ref * (gate_of.repeat_interleave(size, 1) if gate == "head" else gate_of)
        assert float((got[start:start + m].double() - ref).abs().max()) <= 2 ** -8 * float(kv[..., size:].abs().max())
        start += m


@pytest.mark.parametrize("size,page", [(128, 16), (64, 128)])
@pytest.mark.parametrize("ctx,at", [(0, 64), (0, 127), (48, 200), (37, 130), (64, 64)])
def test_values_that_are_not_finite_reach_no_block_before_theirs(size, page, ctx, at):
    """A row is done once the blocks of 64 keys that it sees are added up: an infinite value at position `at` leaves the rows of
    earlier blocks as they are (where 16 rows do not cross into another block, also the rest is the other kernel's)."""
    lens, heads = [(ctx, 300)], 2
    q, cache, bt, step = prompts_over_rows(lens, size, heads, 1, page, ctx + at)
    clean, got, want = torch.zeros_like(q), torch.zeros_like(q), torch.zeros_like(q)
    args = (bt, step, heads, 1, size)
    ops.sink_attention_rows(q, clean, cache, *args, size ** -0.5, None, page, True, None)
    cache[int(bt[0, at // page]), 0, at % page, size:] = float("inf")
    ops.sink_attention_rows(q, got, cache, *args, size ** -0.5, None, page, True, None)
    ops.sink_attention_mma(q, want, cache, *args, size, None, 0, size ** -0.5, None, None, None, None, page)
    before = at // 64 * 64 - ctx
    assert before <= 0 or torch.equal(got[:before], clean[:before])
    if ctx % 16 == 0:
        assert torch.equal(got.isfinite(), want.isfinite()) and torch.equal(got.nan_to_num(), want.nan_to_num())


@pytest.mark.parametrize("m,n,k", [(17, 4, 4), (64, 130, 36), (65, 1664, 260), (66, 1800, 264), (200, 1700, 520), (400, 1300, 2048), (257, 2500, 300)])
def test_products_of_32_bits_in_tiles(m, n, k):
    """One to four CTAs an SM, slices that are short or empty, rows and features that are not there (whose neighbours in memory
    are not finite): bit for bit what the kernel for any operands gives."""
    torch.manual_seed(m + n + k)
    a, w = torch.full((m + 40, k), float("nan"), device="cuda"), torch.full((n + 140, k), float("nan"), device="cuda")
    a[:m], w[:n] = torch.randn(m, k, device="cuda"), torch.randn(n, k, device="cuda")
    got = torch.full((m + 1, n + 3), 7.0, device="cuda")
    ops.gemm_simt(a[:m], w[:n], got[:m, :n])
    odd = torch.empty(m * (k + 1), device="cuda").view(m, k + 1)[:, 1:]
    odd.copy_(a[:m])
    want = torch.empty(m, n, device="cuda")
    ops.gemm_simt(odd, w[:n], want)
    assert torch.equal(got[:m, :n], want)
    assert bool((got[m] == 7).all()) and bool((got[:, n:] == 7).all())


@pytest.mark.parametrize("m,n,k", [(17, 2048, 16), (300, 2048, 64), (65, 8200, 72), (1100, 300, 100), (200, 2050, 260), (70, 32000, 256), (513, 4100, 516)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_products_of_32_bits_in_whole_tiles(m, n, k, dtype):
    """Tiles that one CTA sums, slice after slice (few inputs, or many tiles): bit for bit the kernel for any operands."""
    torch.manual_seed(m + n + k)
    a, w = torch.randn(m, k, device="cuda"), torch.randn(n, k, device="cuda")
    got = torch.full((m + 1, n + 3), 7.0, device="cuda", dtype=dtype)
    ops.gemm_simt(a, w, got[:m, :n])
    odd = torch.empty(m * (k + 1), device="cuda").view(m, k + 1)[:, 1:]
    odd.copy_(a)
    want = torch.empty(m, n, device="cuda", dtype=dtype)
    ops.gemm_simt(odd, w, want)
    assert torch.equal(got[:m, :n], want)
    assert bool((got[m] == 7).all()) and bool((got[:, n:] == 7).all())


@pytest.mark.parametrize("m", [1, 2, 3, 4])
@pytest.mark.parametrize("n,k", [(1, 4), (255, 2052), (1184, 260), (1185, 260), (2500, 36), (5504, 100)])
def test_products_of_32_bits_of_few_rows(m, n, k):
    """Eight and sixteen features a CTA: bit for bit the kernel for any operands; rows that are not there are not read."""
    torch.manual_seed(m + n + k)
    a, w = torch.full((m + 3, k), float("nan"), device="cuda"), torch.randn(n, k, device="cuda")
    a[:m] = torch.randn(m, k, device="cuda")
    got = torch.full((m + 1, n + 3), 7.0, device="cuda")
    ops.gemm_simt(a[:m], w, got[:m, :n], constant_w=True)
    odd = torch.empty(m * (k + 1), device="cuda").view(m, k + 1)[:, 1:]
    odd.copy_(a[:m])
    want = torch.empty(m, n, device="cuda")
    ops.gemm_simt(odd, w, want)
    assert torch.equal(got[:m, :n], want)
    assert bool((got[m] == 7).all()) and bool((got[:, n:] == 7).all())


@pytest.mark.parametrize("kind", ["rows", "latent"])
def test_a_captured_portion_runs_the_kernel_that_its_context_wants(kind, tmp_path, monkeypatch):
    """Equal portions of lone prompts, first at their beginning until one is captured, then far behind: the step there does not
    replay what was captured for the beginning."""
    import kerirax_tiny as kx
    from fastllm_py_b200 import Model, StepEntry

    mixer = kx.pair(kx.left(16, 4, 128, 128, rot=16), kx.right(40, 16, 8, 4)) if kind == "rows" else kx.latent(16, 16, 64, 16, 512, 24)
    raw = kx.config([(mixer, kx.dense(48))], vocab=97, width=40)
    model = Model.load(kx.write(raw, kx.weights(raw, seed=2), tmp_path / "m"), dtype="bfloat16", page_size=16, max_tokens=16384,
                       max_requests=4, max_batched_tokens=2048, max_model_len=4096, cuda_graph=True)
    engine, portion, launched = model.engine, 8 if kind == "rows" else 64, []
    for name in ("sink_attention_rows", "sink_attention_mma", "latent_prompt", "latent_attention_tc"):
        monkeypatch.setattr(ops, name, lambda *a, _f=getattr(ops, name), _n=name, **kw: (launched.append(_n), _f(*a, **kw))[1])
    near, far = ("sink_attention_mma", "sink_attention_rows") if kind == "rows" else ("latent_attention_tc", "latent_prompt")
    tokens = [i % 97 for i in range(4000)]

    def run(rid, at):
        engine.begin(rid)
        if at:
            engine.step([StepEntry(rid, tokens[:at // 2], [])])
            engine.step([StepEntry(rid, tokens[at // 2:at], [])])
        launched.clear()
        out = engine.step([StepEntry(rid, tokens[at:at + portion], [portion - 1])]).clone()
        engine.end(rid)
        return out, list(launched)

    beginning = [run(f"a{i}", 0) for i in range(5)]
    assert [names for _, names in beginning] == [[near]] * 3 + [[]] * 2          # (two eager, one captured, two replayed)
    behind = [run(f"b{i}", 3000) for i in range(5)]
    assert [names for _, names in behind] == [[far]] * 3 + [[]] * 2
    for group in (beginning, behind):
        assert all(torch.equal(out, group[0][0]) for out, _ in group)
    engine.check_status()


@pytest.mark.parametrize("rank,rot", [(64, 64), (128, 64), (256, 128), (256, 192), (512, 0)])
@pytest.mark.parametrize("window", [None, 70])
def test_latent_prompts_of_every_width(rank, rot, window):
    """Queries that arrive in memory of their own (rows of up to seven pieces of 64) and in the later tiles' (eight), one tile and
    several: bit for bit the kernel for single tokens."""
    torch.manual_seed(rank + rot)
    heads, page, width, lens = 16, 16, rank + rot, [(0, 5), (150, 9), (33, 40), (0, 200), (7, 1)]
    per = [-(-(c + m) // page) for c, m in lens]
    bt = torch.zeros(len(lens), max(per), dtype=torch.int32, device="cuda")
    order = torch.randperm(sum(per), device="cuda").to(torch.int32)
    for r, k in enumerate(per):
        bt[r, :k] = order[sum(per[:r]):sum(per[:r]) + k]
    cache = torch.randn(sum(per), page, width, device="cuda").to(torch.bfloat16)
    starts = [sum(m for _, m in lens[:r]) for r in range(len(lens) + 1)]
    n = starts[-1]
    tok_req, positions = i32([r for r, (_, m) in enumerate(lens) for _ in range(m)]), i32([c + i for c, m in lens for i in range(m)])
    q = (0.3 * torch.randn(n, heads * width, device="cuda")).to(torch.bfloat16)
    want, got = (torch.zeros(n, heads * rank, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    ops.latent_attention_tc(q, want, cache, bt, tok_req, positions, heads, rank, rot, window, 0.1, page)
    ops.latent_prompt(q, got, cache, bt, i32(starts), i32([c for c, _ in lens]), i32([m for _, m in lens]), heads, rank, rot, window, 0.1, page)
    assert torch.equal(got, want)


@pytest.mark.parametrize("dim,slabs", [(100, 2), (513, 6), (1028, 1), (2048, 9), (2050, 16), (4096, 11), (8192, 5), (12256, 3)])
@pytest.mark.parametrize("shift", [0, 1])
def test_norm_add_norm_of_partial_sums(dim, slabs, shift):
    """Slabs in one batch and in several, chunks of a thread, rows over several groups of threads, accesses of 16 bytes and of one
    element: the bits of the slabs added in order, rounded, and normed; `out` against float64 within its rounding (2^-9)."""
    torch.manual_seed(dim + slabs)
    rows, ld = 3, dim + 4
    data = torch.empty(slabs * rows * ld + 1, device="cuda")[shift:shift + slabs * rows * ld].view(slabs, rows, ld)
    data.copy_(torch.randn(slabs, rows, ld, device="cuda"))
    partial = SimpleNamespace(data=data, splits=slabs, split_stride=rows * ld, ld=ld, check=lambda: None)
    wa, wb = (1 + 0.2 * torch.randn(2, dim, device="cuda")).to(torch.bfloat16)
    x = torch.randn(rows, dim, device="cuda")
    y = torch.zeros(rows, dim, device="cuda")
    for z in range(slabs):
        y += data[z, :, :dim]
    y = y.to(torch.bfloat16)
    got_x, want_x = x.clone(), x.clone()
    got, want = (torch.empty(rows, dim, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    ops.sandwich_norm_partial(got_x, partial, wa, 1e-5, wb, 1e-6, got)
    ops.sandwich_norm(want_x, y, wa, 1e-5, wb, 1e-6, want)
    assert torch.equal(got_x, want_x) and torch.equal(got, want)
    yd = y.double()
    total = x.double() + yd / torch.sqrt((yd * yd).mean(-1, keepdim=True) + 1e-5) * wa.double()
    ref = total / torch.sqrt((total * total).mean(-1, keepdim=True) + 1e-6) * wb.double()
    assert float(((got.double() - ref).abs() / ref.abs().clamp_min(1e-3)).max()) <= 2 ** -8   # (2^-9, and sums of 32 bits)
