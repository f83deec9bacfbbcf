# SPDX-License-Identifier: Apache-2.0
"""The library's kernels are the same from build to build."""

from __future__ import annotations

from alloy_b200 import build


def test_kernels_do_not_depend_on_how_the_compiler_split_its_work():
    """Split compilation made 150 of 179 kernels differ between two builds of one source, steps by up to 17 %."""
    assert not [f for f in build.NVCC_FLAGS if "split-compile" in f]
