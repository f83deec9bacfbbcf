# SPDX-License-Identifier: Apache-2.0
"""Where a step's state arrays lie does not change a bit of it: output arrays of their own (copied while the particles are
classified), the input arrays themselves (no copy), one of each, and outputs that share memory with an input (copied one
after the other first)."""

from __future__ import annotations

from types import SimpleNamespace

import numpy as np
import pytest
import torch

from alloy_b200.solvers.sph import SolverDFSPH
from alloy_b200.solvers.sph.build import add_fluid_block, add_particle_box
from alloy_b200.solvers.sph.model import ModelBuilder
from alloy_b200.solvers.sph.testing import benchmark_config

pytestmark = pytest.mark.gpu


def _step(cuda, kind):
    cfg = benchmark_config(0.01)
    b = ModelBuilder(gravity=(0.0, 0.0, -9.81))
    b.begin_world()
    add_fluid_block(b, cfg, (0.0, 0.0, 0.0), (9, 7, 11), jitter=0.02, seed=3)
    add_particle_box(b, cfg, (0.0, 0.0, 0.0), (0.13, 0.07, 0.12), open_top=True)
    b.end_world()
    m = b.finalize(cuda)
    n = m.particle_count
    sol = SolverDFSPH(m, cfg)
    s = m.state()
    pool = torch.zeros((4 * n, 3), device=cuda)
    q, qd = pool[:n], pool[n:2 * n]
    q.copy_(s.particle_q)
    qd.copy_(s.particle_qd)
    out = {"apart": (pool[2 * n:3 * n], pool[3 * n:]), "in place": (q, qd), "q in place": (q, pool[2 * n:3 * n]),
           "qd in place": (pool[2 * n:3 * n], qd), "qd over q": (pool[2 * n:3 * n], q)}[kind]
    sol.step(SimpleNamespace(particle_q=q, particle_qd=qd), SimpleNamespace(particle_q=out[0], particle_qd=out[1]), None,
             None, 1.0e-3)
    torch.cuda.synchronize()
    return out[0].cpu().numpy(), out[1].cpu().numpy()


@pytest.mark.parametrize("kind", ["in place", "q in place", "qd in place", "qd over q"])
def test_state_arrays(cuda, kind):
    want, got = _step(cuda, "apart"), _step(cuda, kind)
    assert np.abs(want[1]).max() > 0.0
    for x, y in zip(want, got):
        np.testing.assert_array_equal(x, y)
