"""Kernels that may start while the one before them in the stream still runs
read what their call has written (sorted records, work items, bookmarks, ranks,
job and base tables) by plain loads: __ldg, the non-coherent load, is for memory
that nobody writes while the kernel lives.  Checked in the sources."""
import os
import re

import pytest

from helpers import ROOT

CSRC = os.path.join(ROOT, "ska-gpu-grid_gb300", "csrc")
# arrays in the call's workspace, as the sources name them
WRITTEN = re.compile(r"\b(idx|items|bm|bookmarks|rank|counts|block_off|kept_pos|base|vis_base|"
                     r"tile_base|jobs|nitems|desc|vstride)\b")


def overlapped_sources():
    return sorted(f for f in os.listdir(CSRC)
                  if f.endswith(".cu") and "launch_overlapped(" in open(os.path.join(CSRC, f)).read())


def ldg_arguments(text):
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"__ldg\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        yield text[m.end():i - 1]


def test_the_sources_are_the_expected_ones():
    assert {"gg_bin.cu", "gg_regtile.cu", "gg_gathertile.cu"} <= set(overlapped_sources())


@pytest.mark.parametrize("name", overlapped_sources())
def test_no_noncoherent_load_of_what_the_call_writes(name):
    text = open(os.path.join(CSRC, name)).read()
    # launched plainly, after everything before it has ended
    text = re.sub(r"zero_jobs_kernel\(.*?\n}", "", text, flags=re.S)
    bad = [a for a in ldg_arguments(text) if WRITTEN.search(a)]
    assert not bad, bad
