"""Block sizes of the space-kernel candidates (agdeblend_b200/csrc/engine.cuh,
space_cases): the adjoint kernels reduce the largest |x|^2 over a block by
whole warps, so a block of another size would lose the values of its last
threads."""
import os
import re

from conftest import ROOT

SOURCE = os.path.join(ROOT, "agdeblend_b200", "csrc", "engine.cuh")


def test_candidate_blocks_are_whole_warps():
    with open(SOURCE) as f:
        found = re.findall(r"\badd_(?:fwd|adj)(?:_rows|_pipe)?<([\d, ]+)[^>]*>\(c\)", f.read())
    threads = [int(args.split(",")[4]) for args in found]  # D, P0, P1, P2, threads
    assert len(threads) > 50
    assert [n for n in threads if n % 32 or not 32 <= n <= 1024] == []
