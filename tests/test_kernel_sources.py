"""Rules of the kernels that cannot be shown by running them without hanging a GPU: read from their sources."""
import glob
import os
import re

import pytest

import helpers

CSRC = os.path.join(helpers.PKG_DIR, "csrc")
SOURCES = sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def plain(path):
    """The source without comments and string contents."""
    text = re.sub(r"//[^\n]*", "", open(path).read())
    return re.sub(r"/\*.*?\*/", "", text, flags=re.S)


def kernels(text):
    """(name, body) of every __global__ function."""
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*\)\s*)?(\w+)\s*\(", text):
        at, depth = text.index("{", m.end()), 0
        for i in range(at, len(text)):
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            if depth == 0:
                yield m.group(1), text[at:i]
                break


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_tensor_memory_is_taken_before_successors_may_start(path):
    """A successor that is placed beside a CTA without its columns yet could take them and wait for this grid for good. A trigger
    before the allocation is allowed where the CTA leaves right after it."""
    for name, body in kernels(plain(path)):
        alloc = re.search(r"\btmem_alloc\w*\(", body)
        for m in re.finditer(r"\bpdl_trigger\(\);", body[:alloc.start()] if alloc else ""):
            assert "return;" in body[m.end():body.index("}", m.end())], name
