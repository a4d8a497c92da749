"""Rules that a wrong kernel would break without a wrong result, or by a hang or a read out of range: checked on the
kernels' sources, since no run may provoke them."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "fastllm-py_b200" / "csrc"


def test_cuda_core_attention_looks_up_only_pages_in_sight():
    """A window's pages go back to the pool when every window has passed them, and the table then has -1 in their place: a
    tile's rows below the first key in sight must not look theirs up, however they are copied."""
    text = (CSRC / "attention_simt.cu").read_text()
    lookups = [m.start() for m in re.finditer(r"\bbt\[", text)]
    assert lookups
    for at in lookups:
        guard = text[text.rindex("if (", 0, at):at].split("{")[0]
        assert "j >= first" in guard and "r < keys" in guard, guard


def waits_on_values(name):
    """The o_done protocol of an attention kernel on the tensor cores, from its source: how many barriers, which one a
    block's value product arrives on, and the waits (barrier, parity) of the warps that rescale and read the accumulators:
    [one in every block, if there is one], where they rescale, at the end; functions of the block i, or of their number n."""
    text = (CSRC / name).read_text()
    expr = lambda c: re.sub(r"(\d)u\b", r"\1", c.replace("(uint32_t)", "").replace("n_tiles", "n").replace("n_blocks", "n"))
    index = lambda c: expr(c[len("&o_done["):-1]) if "[" in c else "0"
    commit = re.search(r"commit\((&o_done\[[^\]]*\]|o_done)\)", text).group(1)
    commit = index(commit).replace("b", "(i & 1)")
    waits = [(index(m.group(1)), expr(m.group(2))) for m in
             re.finditer(r"warp_wait\((&o_done\[[^\]]*\]|o_done), (.*?), abort_flag\)", text)]
    return commit, waits


@pytest.mark.parametrize("name", ["latent_attention_tc.cu", "attention_prefill_tc.cu"])
def test_waits_for_the_value_products_cannot_pass_early(name):
    """A wait on a barrier's parity is over when the phase of that parity is the one completed last: also while the barrier
    still is two phases behind.  Every state that the value products can be in at each wait, going only by what the warp
    itself has waited for, with every choice of the blocks that rescale: a wait is over exactly when its product is done."""
    commit, waits = waits_on_values(name)
    assert 2 <= len(waits) <= 3
    every, rescale, final = ([None] + waits)[-3:]
    at = lambda e, **v: eval(e, {}, v)                                    # the source's own expressions
    barrier_of = lambda t: at(commit, i=t)

    def wait(known, most, target, barrier, parity):
        """`known` .. `most` products may be done, in order; waits for product `target`."""
        for done in range(known, most + 1):
            phase = sum(barrier_of(t) == barrier for t in range(done))    # phases of this barrier that are complete
            assert ((phase - 1) & 1 == parity) == (done > target), (done, target)
        return max(known, target + 1)

    for n in range(1, 9):
        for choice in range(1 << n):
            known = 0                                                     # so many products are known to be done
            for i in range(n):                                            # product i waits for this warp: at most i are done
                if every is not None and i > 1:
                    known = wait(known, i, i - 2, at(every[0], i=i), at(every[1], i=i))
                if i > 0 and choice >> i & 1:
                    known = wait(known, i, i - 1, at(rescale[0], i=i), at(rescale[1], i=i))
            wait(known, n, n - 1, at(final[0], n=n), at(final[1], n=n))


def test_epilogue_warps_give_up_together():
    """The epilogue's four warps meet at barriers of their own, so they must leave a unit of work together.  The abort flag can
    change between two warps' looks at it: no decision to leave may be a look after a barrier, only the barrier's own vote."""
    for path in sorted(CSRC.glob("*.cu")):
        text = path.read_text()
        assert not re.search(r"epilogue_sync\(\);[^\n]*\n[^\n]*abort_flag", text), path.name
        voted = re.findall(r"epilogue_any\([^;]*abort_flag", text)
        assert len(voted) == {"gemm_tcgen05.cu": 3, "moe.cu": 1}.get(path.name, 0), path.name
    assert re.search(r"epilogue_any\(bool flag\).*?red\.or\.pred", (CSRC / "tcgen05.cuh").read_text(), re.S)


def test_a_pair_tile_has_one_width():
    """The box of the token rows, the bytes that a stage expects and the MMA's N all follow the width of a CTA pair's tiles: it
    is worked out in one place, which also makes the map."""
    text = (CSRC / "gemm_tcgen05.cu").read_text()
    assert len(re.findall(r"\btc_pair_tile_tokens\(", text)) == 2                     # the function and its one call
    launch = text[text.index("static int launch_tc_pair("):]
    launch = launch[:launch.index("\n}\n")]
    assert "tc_pair_tile_tokens(" in launch and "make_map(&map_a, A, M, K, lda, wt / 2)" in launch


@pytest.mark.parametrize("name, kernels", [("gemm_tcgen05.cu", ["gemm_tc_kernel", "gemm_tc_pair_kernel"]), ("moe.cu", ["moe_group_kernel"])])
def test_products_that_give_up_wait_for_their_copies(name, kernels):
    """A CTA that leaves with copies on their way would have them land in the next CTA's shared memory: after all roles have
    met, the thread that issued every fill waits for them, where the abort flag is set, before the CTA (or the pair) may go."""
    text = (CSRC / name).read_text()
    for kernel in kernels:
        body = text[text.index(f" {kernel}("):]
        body = body[:body.index("\n}\n")]
        met = body.rindex("tc_fence_before();\n    __syncthreads();")
        drain = body.index("if (threadIdx.x == 0 && *abort_flag) tma_drain(full_bar, ", met)
        assert drain < body.index("dealloc", met) and ("cluster_sync_all" not in body or drain < body.index("cluster_sync_all", met))
        ring = body[body.index("int issued = 0;"):met]
        assert ring.count("++issued;\n") == 1 and ring.index("++issued;") < ring.index("if (++s ==")


@pytest.mark.parametrize("name", ["latent_attention_tc.cu", "attention_prefill_tc.cu"])
def test_attention_that_gives_up_waits_for_its_copies(name):
    """The same in the attention kernels: the producer, where the abort flag is set, waits for the rings' fills and for the
    queries, with waits that the flag does not cut short."""
    text = (CSRC / name).read_text()
    drain = re.search(r"if \(\*abort_flag\) \{[^}]*?for \(int k = max\(0, i - \w+\); k < i; \+\+k\)[^}]*\}", text).group(0)
    filled = set(re.findall(r"expect(?:_tx)?\(&?(\w+)", text)) - {"uint64_t"}                # (not the wrapper itself)
    assert filled and all(re.search(rf"wait\(&?{bar}\b[^;]*never\)", drain) for bar in filled), (filled, drain)
