"""Rules that a wrong kernel would break without a wrong result, or by a hang or a read out of range: checked on the
kernels' sources, since no run may provoke them."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "fastllm-py_b200" / "csrc"


def test_cuda_core_attention_looks_up_only_pages_in_sight():
    """A window's pages go back to the pool when every window has passed them, and the table then has -1 in their place: a
    tile's rows below the first key in sight must not look theirs up, in either way of copying them."""
    text = (CSRC / "attention_simt.cu").read_text()
    lookups = [m.start() for m in re.finditer(r"\bbt\[", text)]
    assert len(lookups) == 2
    for at in lookups:
        guard = text[text.rindex("if (", 0, at):at].split("{")[0]
        assert "j >= first" in guard and "r < keys" in guard, guard
