"""Shared memory that threads write and bulk copies then read or overwrite is
accessed through two proxies: a proxy fence has to stand between, or the two are
unordered. No run shows a missing one reliably, so the sources are read."""
import os
import re

import pytest

from conftest import ROOT


def body(unit, name):
    """Code of a function of csrc/<unit>, without comments."""
    with open(os.path.join(ROOT, "hornofusion-full3d_b200", "csrc", unit)) as f:
        code = re.sub(r"//[^\n]*", "", f.read())
    start = code.index("{", re.search(rf"\b{name}\([^;{{]*\)\s*{{", code).start())
    depth, at = 1, start + 1
    while depth:
        depth += {"{": 1, "}": -1}.get(code[at], 0)
        at += 1
    return code[start:at]


# (unit, function, generic accesses, what makes them visible to the issuing thread)
HAND_OVERS = [("tdma.cu", "load_lines", r"write_line<", r"__syncwarp\(\)"),
              ("tdma.cu", "tdma_factor_kernel", r"factor_line<", r"__syncwarp\(\)"),
              ("tdma.cu", "tdma_old_kernel", r"r\[kOEnd \* K\] = ", r"__syncthreads\(\)"),
              ("cg_dsm.cu", "push_allsum", r"st_shared_f64", r"__syncthreads\(\)")]


@pytest.mark.parametrize("unit,name,access,sync", HAND_OVERS)
def test_fence_between_accesses_and_bulk_copies(unit, name, access, sync):
    code = body(unit, name)
    assert re.search(access + r"(?:(?!" + sync + r").)*?(?:fence_proxy_async\(\)|"
                     r"fence\.proxy\.async)(?:(?!" + access + r").)*?" + sync, code, re.S)
