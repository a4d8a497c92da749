"""How the decode kernel's keys are split, with sequences of unequal lengths."""
from types import SimpleNamespace

import pytest

from fastllm_py_b200.native.attention import decode_split_keys


@pytest.mark.parametrize("n,kv_heads,longest", [(1, 16, 1), (1, 16, 513), (8, 32, 2049), (64, 8, 1258), (24, 16, 1442), (200, 1, 70000)])
def test_split_of_unequal_lengths(n, kv_heads, longest):
    equal = decode_split_keys(n, kv_heads, longest)
    assert decode_split_keys(n, kv_heads, longest, mean_seq_len=longest) == equal
    assert decode_split_keys(n, kv_heads, longest, mean_seq_len=10 * longest) == equal       # (a mean cannot exceed the longest)
    for mean in (1, longest // 3 + 1, longest // 2 + 1):
        keys = decode_split_keys(n, kv_heads, longest, mean_seq_len=mean)
        assert keys % 64 == 0 and 64 <= keys <= 1024
        stretch = -(-mean // 256) * 256                     # one answer for all means of a stretch of 256
        assert keys == decode_split_keys(n, kv_heads, longest, mean_seq_len=stretch) \
            == decode_split_keys(n, kv_heads, longest, mean_seq_len=max(1, stretch - 255))


def test_a_prompt_beside_decoding_requests_does_not_lengthen_their_splits(monkeypatch):
    """The plan of a mixed step looks at the requests with one token only."""
    from fastllm_py_b200.native import attention as fast
    from fastllm_py_b200.parts.attention import Attention

    part = object.__new__(Attention)
    part.heads = part.kv_heads = 16
    part.head_dim, part.ctx = 128, SimpleNamespace(device="cpu")
    monkeypatch.setattr(Attention, "_fast", lambda self: fast)
    monkeypatch.setattr(fast, "num_sms", lambda device: 148)
    plans = []
    for extra in ([], [(0, 488)], [(1500, 450)]):
        lens = [(400 + 40 * i, 1) for i in range(24)] + extra
        step = SimpleNamespace(n_decode_tokens=24, for_graph=False, plans={}, ctx_lens=[c for c, _ in lens], q_lens=[q for _, q in lens],
                               max_seq_len=max(c + q for c, q in lens))
        Attention.plan_step(part, step)
        plans.append(step.plans[part.plan_key])
    assert plans[0] == plans[1] == plans[2]
    keys, splits = plans[0]
    assert keys * splits >= 400 + 40 * 23 + 1 and keys * (splits - 1) < 400 + 40 * 23 + 1


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
