"""CPU: the library's device memory is written in the order of its own stream.

The library's stream is created with cudaStreamNonBlocking, so nothing orders
it after work on the default stream, and a copy from pageable memory or a
memset there may still be in flight when the call returns.  The sources
therefore use only the forms that take a stream.
"""
import glob
import os
import re

import pytest

from conftest import ROOT

CSRC = sorted(glob.glob(os.path.join(ROOT, "milc-qphix_b200", "csrc", "*")))
# writes to device memory on the default stream
DEFAULT_STREAM = re.compile(r"\bcudaMemset\s*\(|\bcudaMemcpyToSymbol\s*\(|\bcudaMemcpy\s*\([^;]*HostToDevice", re.S)


@pytest.mark.parametrize("path", CSRC, ids=os.path.basename)
def test_no_device_write_on_the_default_stream(path):
    text = re.sub(r"//[^\n]*", "", open(path).read())
    assert not DEFAULT_STREAM.findall(text)
