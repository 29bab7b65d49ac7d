"""Kernels launched with programmatic stream serialization (launch_pdl in
agdeblend_b200/csrc/engine.cuh) wait for the kernels before them: each calls
pdl_enter, and no block returns before it, so that a kernel's completion
implies its predecessors'."""
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "agdeblend_b200", "csrc")
# launched by name, and through the tables of kernels of these headers
HEADERS = ["fast.cuh", "plane_dft.cuh", "time_pair.cuh"]


def _kernels(header):
    """name -> body of every __global__ function of a header."""
    with open(os.path.join(CSRC, header)) as f:
        text = f.read()
    out = {}
    nested = r"\((?:[^()]|\((?:[^()]|\([^()]*\))*\))*\)"  # parentheses, three deep
    for m in re.finditer(rf"__global__ void\s+(?:__launch_bounds__{nested}\s*)?"
                         r"(\w+)\([^{;]*\)\s*\{", text):
        depth, end = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        out[m.group(1)] = text[m.end():end]
    return out


def test_kernels_wait_before_they_return():
    with open(os.path.join(CSRC, "engine.cuh")) as f:
        engine = f.read()
    found = {}
    for h in HEADERS:
        found.update(_kernels(h))
    assert {"space_adj_pipe", "plane_dft", "line_dft", "axis_dft", "time_fwd_pair"} <= set(found)
    others = {**_kernels("kernels.cuh"), **_kernels("wavelet_fast.cuh")}
    by_name = set(re.findall(r"launch_pdl\((\w+)<R>", engine)) | {"wavelet_fast"}
    assert {"record_gather", "next_lambda"} <= by_name
    found.update({n: others[n] for n in by_name})
    for name, body in found.items():
        head, wait, _ = body.partition("pdl_enter();")
        assert wait, name
        assert "return" not in re.sub(r"\[&\][^{]*\{[^}]*\}", "", head), name
