"""Index arithmetic of the block copies, compiled for the host and checked without a GPU."""

import os
import shutil

import pytest

from test_host_logic import CSRC, ROOT, _build_and_run  # noqa: F401


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_copies_of_the_largest_32_bit_blocks(tmp_path):
    _build_and_run(tmp_path, "check_copy", [os.path.join(ROOT, "tests", "host", "check_copy.cpp")], [])
