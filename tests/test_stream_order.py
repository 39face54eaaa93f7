"""The library's streams are non-blocking ones, which copies and clears on the
default stream are not ordered with: every one of them names its stream."""
import os
import re

import pytest

from kerrtracecpp2_b200 import build


@pytest.mark.parametrize("src", build.CU_SOURCES + build.CXX_SOURCES)
def test_no_copy_on_the_default_stream(src):
    text = open(os.path.join(build.CSRC, src)).read()
    calls = re.findall(r"\bcuda(?:Memcpy|Memcpy2D|Memset|MemcpyToSymbol|MemcpyFromSymbol)\(", text)
    assert not calls, calls
