"""What the host decides per step: how the decode kernel's keys are split, and which kernel serves prompts."""
from types import SimpleNamespace

import pytest


@pytest.mark.parametrize("lens", [[300 + 37 * i for i in range(64)], [5, 1900], [360 + 45 * i for i in range(24)]])
def test_split_follows_the_longest_sequence_only(lens, monkeypatch):
    """The split decides how a token's sums are rounded, and which captured step runs it: a batch that grows keeps it for 256
    tokens, and the lengths of shorter neighbours do not enter."""
    from fastllm_py_b200.native import attention as fast
    from fastllm_py_b200.parts.attention import Attention

    part = object.__new__(Attention)
    part.heads, part.kv_heads, part.head_dim, part.ctx = 16, 8, 128, SimpleNamespace(device="cpu")
    monkeypatch.setattr(Attention, "_fast", lambda self: fast)
    monkeypatch.setattr(fast, "num_sms", lambda device: 148)

    def plan(ctx_lens):
        step = SimpleNamespace(n_decode_tokens=len(ctx_lens), for_graph=True, plans={}, ctx_lens=ctx_lens, q_lens=[1] * len(ctx_lens),
                               max_seq_len=max(ctx_lens) + 1)
        Attention.plan_step(part, step)
        return step.plans[part.plan_key]

    grown = [plan([c + k for c in lens]) for k in range(1024)]
    assert sum(a != b for a, b in zip(grown, grown[1:])) <= 4
    assert plan(lens) == plan([1] * (len(lens) - 1) + [max(lens)]) == plan([max(lens)] * len(lens))
    keys, splits = plan(lens)
    assert keys == fast.decode_split_keys(len(lens), 8, max(lens) + 1) and keys * splits >= max(lens) + 1


@pytest.mark.parametrize("lens,heads,single,pays", [([(0, 2048)], 16, False, True), ([(1500, 8)], 4, False, True), ([(0, 4)], 16, False, False),
                                                    ([(0, 8)] * 20, 32, False, False), ([(0, 100)] * 8, 32, False, True),
                                                    ([(700, 1)] * 16 + [(0, 4)], 16, False, False), ([(700, 1)] * 16, 16, True, True),
                                                    ([], 16, False, True)])
def test_prompt_attention_over_rows_goes_where_it_is_faster(lens, heads, single, pays):
    """Measured sides of the rule; single tokens count only where the kernel serves them; a step without lengths is accepted."""
    from fastllm_py_b200.native.ops import _sink_rows_pay

    step = SimpleNamespace(q_lens=[q for _, q in lens], ctx_lens=[c for c, _ in lens]) if lens else SimpleNamespace()
    assert _sink_rows_pay(step, heads, single, 148) is pays


@pytest.mark.parametrize("lens,heads,pays", [([(0, 8)] * 20, 16, False), ([(0, 8)] * 20, 32, True), ([(0, 3)] * 60, 32, False), ([(0, 37)] * 8, 32, True),
                                             ([(0, 64)], 16, False), ([(0, 128)], 16, True), ([(1000, 64)], 16, True),
                                             ([(500, 4)] * 16, 16, True), ([(100, 1)] * 140, 16, False)])
def test_latent_prompt_kernel_where_it_is_faster(lens, heads, pays, monkeypatch):
    """Measured sides of the rule for a latent of 512; without the lengths behind, and under capture, the rule by rows."""
    from fastllm_py_b200.parts import latent

    monkeypatch.setattr(latent.ops, "latent_prompt_takes", lambda *a: True)
    monkeypatch.setattr(latent.ops, "sm_count", lambda device: 148)
    part = object.__new__(latent.LatentAttention)
    part.rank, part.rot, part.heads, part.window, part.ctx = 512, 64, heads, None, SimpleNamespace(dtype=None, device=None)
    n = sum(q for _, q in lens)
    step = SimpleNamespace(q_lens=[q for _, q in lens], ctx_lens=[c for c, _ in lens])
    assert part._prompts(step, n, 16) is pays
    rows = 4 * sum(-(-q // 8) for q in step.q_lens) <= n and n * heads // 16 > 148
    assert part._prompts(SimpleNamespace(q_lens=step.q_lens), n, 16) is rows
    step.for_graph = True
    assert part._prompts(step, n, 16) is rows


@pytest.mark.parametrize("kind", ["normed", "sink", "latent"])
def test_the_prompt_kernel_is_part_of_a_captured_steps_key(kind, monkeypatch):
    """Equal portions of a lone prompt are captured: one far behind must not replay the kernel that suited the first.  Decided
    once a step, in its plan."""
    import torch

    from fastllm_py_b200.native import ops
    from fastllm_py_b200.parts import latent, normed_attention, sink_attention

    monkeypatch.setattr(ops, "sm_count", lambda device: 148)
    monkeypatch.setattr(ops, "latent_prompt_takes", lambda *a: True)
    monkeypatch.setattr(ops, "sink_decode_takes", lambda *a: True)
    part = object.__new__({"normed": normed_attention.NormedAttention, "sink": sink_attention.SinkAttention,
                           "latent": latent.LatentAttention}[kind])
    part.ctx = SimpleNamespace(device=torch.device("cuda"), dtype=torch.bfloat16, page_size=16)
    part.heads, part.kv_heads, part.dim, part.vdim, part.window, part.chunk = 16, 4, 128, 128, None, None
    part.keep_first, part.softcap, part.bias_rows, part.rank, part.rot = 0, None, None, 512, 64

    def key(ctx, q):
        step = SimpleNamespace(plans={}, ctx_lens=[ctx], q_lens=[q], max_seq_len=ctx + q, n_tokens=q, n_decode_tokens=0, for_graph=False)
        part.plan_step(step)
        return part.graph_key(step)

    q = 8 if kind != "latent" else 64
    assert key(0, q) != key(3000, q) and key(0, q)[-1] is False
    assert key(3000, q) == key(5000, q) and key(3000, q)[-1] is True
    if kind == "sink":
        part.softcap = 30.0
        capped = part.plan_key
        assert key(3000, q)[-1] is False                      # a layer that the kernel does not serve, with a plan of its own
        part.softcap = None
        assert part.plan_key != capped


@pytest.mark.parametrize("requests,rows", [(65535, True), (65536, False)])
def test_more_tiles_than_a_grid_holds_stay_with_the_other_kernel(requests, rows, monkeypatch):
    """The tiles of 128 tokens are a grid's y, which the other kernel's are not: no step is refused for them."""
    import torch

    from fastllm_py_b200.native import ops

    called = []
    monkeypatch.setattr(ops, "_require_cuda", lambda *a: None)
    monkeypatch.setattr(ops, "sm_count", lambda device: 148)
    monkeypatch.setattr(ops, "sink_attention_rows", lambda *a: called.append(True))
    monkeypatch.setattr(ops, "sink_attention_mma", lambda *a: called.append(False))
    q = torch.empty(64, 256, dtype=torch.bfloat16)
    ops.sink_attention_tc(q, q, torch.empty(4, 1, 16, 256, dtype=torch.bfloat16), None, SimpleNamespace(n_requests=requests), 2, 1, 128, 128,
                          None, 0, 1.0, None, None, None, None, 16)
    assert called == [rows]
