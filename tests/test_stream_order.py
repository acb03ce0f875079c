"""A context works on its own non-blocking stream, which the legacy stream does
not order, and a copy of up to 64 KB from pageable memory may return before it
has landed: the sources use the stream-ordered calls only."""
import glob
import os
import re

import pytest

from conftest import ROOT

SOURCES = sorted(glob.glob(os.path.join(ROOT, "3d-rism-cuda_b200", "csrc", "*.c*")))


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_no_legacy_stream_copies(path):
    legacy = re.compile(r"\bcudaMem(?:cpy|set)(?:[23]D|ToSymbol|FromSymbol)?\s*\(")
    with open(path) as f:
        found = [k for k, line in enumerate(f, 1) if legacy.search(line)]
    assert not found, (os.path.basename(path), found)
