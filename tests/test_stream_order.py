"""The context's streams are not ordered after the legacy default stream.

They are created non-blocking, so a memset or an upload issued there may still
be under way when a kernel of the context starts (a memset of device memory
may return early, an upload from pageable memory once it is staged). Every
one of them therefore names a stream.
"""
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "kessler-syndrom-simulation_b200", "csrc")


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith(".cu")))
def test_no_copy_or_memset_on_the_legacy_stream(name):
    text = open(os.path.join(CSRC, name)).read()
    found = re.findall(r"cudaMem(?:set|cpy)(?:2D|3D|ToSymbol|FromSymbol|Peer)?\s*\(", text)
    assert not found, found
