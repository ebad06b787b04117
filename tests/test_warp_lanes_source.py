"""Warp-synchronous operations name their lanes: by the full mask, a ballot or a
match, never by __activemask(), which does not say which lanes arrive together."""
import os

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mpqpcudasolver_gb300", "csrc")


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".h"))))
def test_no_activemask(name):
    with open(os.path.join(CSRC, name)) as f:
        assert "__activemask" not in f.read()
