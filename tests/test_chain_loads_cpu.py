"""Loads of kernels that are resident while the kernel before them still writes their operands."""

from __future__ import annotations

import re
from pathlib import Path

import pytest

import mini_inference_engine_b200

SOURCES = sorted(Path(mini_inference_engine_b200.__file__).parent.joinpath("csrc").glob("*.cu*"))

# The read-only path is for data that nobody writes during the kernel's lifetime.  A kernel of a launch chain starts
# before its predecessor has written, and only ordinary loads keep their place behind the wait.
READ_ONLY = re.compile(r"__ldg\s*\(|ld\.global(\.\w+)*\.nc\b|const\s+[\w:]+\s*\*\s*(const\s+)?__restrict__")


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_no_read_only_loads(path):
    code = re.sub(r"//[^\n]*", "", path.read_text())
    assert READ_ONLY.findall(code) == []
