"""Dynamic shared memory that 16-byte asynchronous copies write to.

``extern __shared__ double s[]`` only promises 8-byte alignment; where it lies
behind static arrays of mixed sizes, a 16-byte ``cp.async`` into it is
misaligned, a fault, whenever the linker places it on an odd multiple of
eight.  Every dynamic array of a source with such copies states its alignment."""
import glob
import os
import re

import pytest

import bd_b200 as B

SOURCES = sorted(glob.glob(os.path.join(B.PKG, "csrc", "*.cu*")))


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_dynamic_shared_memory_of_16_byte_copies_is_aligned(path):
    text = open(path).read()
    if not re.search(r"cp\.async\.cg\.shared\.global", text):
        return
    arrays = re.findall(r"extern\s+__shared__\s+([^;]*);", text)
    assert all("__align__(16)" in a for a in arrays), arrays
