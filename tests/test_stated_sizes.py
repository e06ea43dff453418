"""The size of the allocation-free entry point's array, wherever it is stated."""
import os
import re

import pytest

from helpers import ROOT

SOURCE = os.path.join("ska-gpu-grid_gb300", "csrc", "gg_noalloc.cu")


def size():
    with open(os.path.join(ROOT, SOURCE)) as f:
        return int(re.search(r"static_assert\(kScratchBytes == (\d+)", f.read()).group(1))


@pytest.mark.parametrize("name", [os.path.join("include", "gg.h"), "INTEGRATION.md", SOURCE])
def test_the_stated_size_is_the_array_s(name):
    with open(os.path.join(ROOT, name)) as f:
        text = " ".join(f.read().split())
    stated = re.findall(r"([\d,]{7,}) bytes[^()]{0,8}[,(] ?(\d+\.\d) MiB", text)
    assert stated
    for number, mib in stated:
        assert int(number.replace(",", "")) == size() and float(mib) == round(size() / 2**20, 1)
