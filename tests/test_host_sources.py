"""The host sources compile for any host that CUDA runs on: no architecture's intrinsics in them."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "neonengine_b200", "csrc")


@pytest.mark.parametrize("name", sorted(os.listdir(CSRC)))
def test_no_host_intrinsics(name):
    with open(os.path.join(CSRC, name)) as f:
        found = re.findall(r"\w*intrin\.h|arm_neon\.h|\b__m\d+\w*|\b_mm\d*_\w+", f.read())
    assert not found, found
