"""What a kernel may rely on when it is launched before the kernel ahead of it has ended, read from the sources."""

from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "forge_engine_b200" / "csrc"
SOURCES = sorted(CSRC.glob("*.cu*"))


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_no_launch_switches_a_wait_off(path):
    """What earlier kernels wrote is visible only to a grid that executes griddepcontrol.wait itself: that some kernel in
    between has waited is not enough.  So no field of the launch's parameters takes a wait out."""
    text = re.sub(r"//[^\n]*", "", path.read_text())
    assert not re.search(r"if\s*\(\s*!\s*p\.\w+[^;{}]*\)\s*\{?\s*pdl_wait\(\)", text)
    assert not re.search(r"waited\s*=\s*!?\s*p\.", text)
