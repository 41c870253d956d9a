"""Kernels that are set up while their producer still runs (launch_behind):
each waits for it first, and reads what it writes by plain loads.  The
read-only path (__ldg, const __restrict__) is for data that is constant for
the kernel's whole life, which a producer's output here is not.  Read from the
sources: no run can show a load that the compiler was merely allowed to move."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gc-fg_gb300", "csrc")
SRC = {f: open(os.path.join(CSRC, f)).read() for f in sorted(os.listdir(CSRC)) if f.endswith((".cu", ".cuh"))}
TEXT = "\n".join(SRC.values())
# what a kernel of such a chain writes for the next one: histograms, t-link
# tables, per-image states, and the solver's arena
PRODUCED = r"(?:hist|hf|hb|lut|tl_lut|ist|hfin|reach|cap|exc|h|tmask|tile_pos|tile_act)"
KERNELS = sorted(set(re.findall(r"launch_behind\((k_\w+)", TEXT)))


def _function(name):
    """(parameter list, body) of the kernel or device function `name`."""
    m = re.search(r"\b%s\s*\(((?:[^()]|\([^()]*\))*)\)\s*\{" % name, TEXT)
    depth, i = 1, m.end()
    while depth:
        depth += {"{": 1, "}": -1}.get(TEXT[i], 0)
        i += 1
    return m.group(1), TEXT[m.end():i]


def test_the_kernels_are_found():
    assert {"k_tlut_b", "k_build_img_b", "k_extract_rows"} <= set(KERNELS)


@pytest.mark.parametrize("name", KERNELS)
def test_waits_first(name):
    _, body = _function(name)
    before = body.split("cudaGridDependencySynchronize();")
    assert len(before) == 2
    assert not re.search(r"=|__ld", re.sub(r"constexpr [^;]*;", "", before[0]))  # declarations only


@pytest.mark.parametrize("name", KERNELS + ["build_strip"])
def test_reads_the_producer_by_plain_loads(name):
    params, body = _function(name)
    assert not re.search(r"__ldg\(\s*(?:\w+(?:\.|->))?%s\b" % PRODUCED, body)
    assert not re.search(r"const\s+\w+\s*\*\s*__restrict__\s+%s\b" % PRODUCED, params)
