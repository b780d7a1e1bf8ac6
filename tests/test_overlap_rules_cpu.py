"""Rules of the kernels that overlap their predecessor (plqcd_b200/csrc/pdl.cuh),
read from the sources: the launch dependency is waited for before the first
access to memory and before any way out of the kernel. A read ahead of the wait
may see what the predecessor's predecessor left; a block that leaves without it
lets its grid complete before the one it follows."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "plqcd_b200", "csrc")
OVERLAPPED = ["k_cg_p_x", "k_dslash_ahead", "k_dslash_mrhs_pair_ahead", "k_hop_sum_finish", "k_mrhs_links_f64"]
# a way out; a dereference; a load, store, copy or atomic by name
FORBIDDEN = r"\breturn\b|->|\*\s*[\w.]*\bhalt\b|\b\w*(?:load|store|ld_|issue_|atomic|cp_async)\w*\s*(?:<[^;()]*>)?\("


def _kernels():
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\(", text):
            start = text.index("{", m.end())
            depth, end = 1, start + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            out[m.group(1)] = text[start:end]
    return out


def test_overlapped_kernels_are_the_known_ones():
    assert sorted(k for k, body in _kernels().items() if "pdl_start()" in body) == OVERLAPPED


@pytest.mark.parametrize("name", OVERLAPPED)
def test_nothing_precedes_the_wait(name):
    before = _kernels()[name].split("pdl_start()")[0]
    assert not re.findall(FORBIDDEN, before)


@pytest.mark.parametrize("name", OVERLAPPED)
def test_reads_are_ordinary_loads(name):
    """Fields that a predecessor may have written don't come through the
    non-coherent path, whose loads may move ahead of the wait (the formats'
    own load functions take it)."""
    assert not re.findall(r"__ldg|ld\.global\.nc|\w*IO(?:<[^>]*>)?::load(?:_raw)?\s*\(", _kernels()[name])
