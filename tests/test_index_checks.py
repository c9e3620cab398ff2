"""Every index into the arrays that the bounds-checked build covers goes through YAMC_IX, reads as well
as writes: a scan of the kernels' source (a lane's own place, `lane` plus a constant, needs no check)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "yamc_b200", "csrc")


def _unchecked(text, arrays):
    uses = re.findall(r"\b(?:%s)\[(?!YAMC_IX|(?:\d+ \+ )?lane\])[^\]]*\]" % "|".join(arrays), text)
    return [u for u in uses if not re.match(r"\w+\[(k\w+|[\w/ ]+kBlk)\]$", u)]


def _part(name, begin, end):
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    a = text.index(begin)
    return text[a:text.index(end, a)]


def test_pair_filter_of_the_chain_kernel():
    text = _part("yamc_chain.cuh", "__device__ __forceinline__ void real_part(", "__device__ __noinline__ void real_part_forces(")
    assert "queue[YAMC_IX" in text and "blocks[YAMC_IX" in text and "nb[YAMC_IX" in text
    assert _unchecked(text, ["atom_s", "meta_s", "blocks", "nb", "queue"]) == []


def test_whole_configuration_sums():
    text = _part("yamc_sums.cuh", "k_real_energy(", "// k space along the rows of the k grid")
    assert _unchecked(text, ["order", "list", r"queue\[warp\]"]) == []
    text = _part("yamc_sums.cuh", "k_rho_rows(", "// radial distribution functions")
    assert _unchecked(text, ["alist", "out"]) == []
