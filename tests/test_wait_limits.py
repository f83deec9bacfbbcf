# SPDX-License-Identifier: Apache-2.0
"""One default limit of the solves' barrier waits: the library's (include/alloy_dfsph.h), which ``barrier_wait()`` without
arguments restores."""

from __future__ import annotations

import inspect
import re
from pathlib import Path

from alloy_b200 import _lib
from alloy_b200.solvers.sph import SolverDFSPH

ROOT = Path(__file__).resolve().parents[1]


def test_barrier_wait_restores_the_library_default():
    header = (ROOT / "include" / "alloy_dfsph.h").read_text()
    bits = re.search(r"#define ADF_BARRIER_POLLS \(1ll << (\d+)\)", header)
    assert bits and _lib.ADF_BARRIER_POLLS == 1 << int(bits.group(1))
    p = inspect.signature(SolverDFSPH.barrier_wait).parameters
    assert p["polls"].default == _lib.ADF_BARRIER_POLLS
    assert p["extra_arrivals"].default == 0
    source = (ROOT / "alloy_b200" / "csrc" / "dfsph_capi.cu").read_text()
    assert re.search(r"persist_wait = ADF_BARRIER_POLLS;", source)
