# SPDX-License-Identifier: Apache-2.0
"""Which form a solve's one launch takes at the sizes on both sides of each limit (of a device of 148 SMs), and that a step
does take it: fewer launches than one kernel per phase."""

from __future__ import annotations

import pytest
import torch

from alloy_b200.solvers.sph import SolverDFSPH
from alloy_b200.solvers.sph.testing import dam_break

pytestmark = pytest.mark.gpu
SMALL, DEEP, WIDE = 0, 1, 2


@pytest.mark.parametrize("counts,form,threads", [
    ((1, 1, 1), SMALL, 256),
    ((33, 33, 34), SMALL, 256),   # 37,026 of 37,888
    ((33, 34, 34), DEEP, 288),    # 38,148
    ((53, 53, 53), DEEP, 1024),   # 148,877 of 151,552
    ((54, 54, 54), WIDE, 640),    # 157,464
    ((57, 57, 58), WIDE, 640),    # 188,442 of 189,440: one round against two
    ((58, 58, 58), DEEP, 1024),   # 195,112: two rounds either way
])
@pytest.mark.parametrize("solver", ["jacobi", "cg"])
def test_form_by_size(cuda, counts, form, threads, solver):
    if torch.cuda.get_device_properties(cuda).multi_processor_count != 148:
        pytest.skip("the sizes are those of 148 SMs")
    box = tuple(0.01 * (c + 2) for c in counts)
    launches = []
    for one_launch in (True, False):
        sc = dam_break(counts=counts, box=box, spacing=0.01, dt=5.0e-4, device=cuda, pressure_solver=solver)
        sol = SolverDFSPH(sc.model, sc.config)
        sol.autotune(False)
        sol.use_graphs(False)
        if not one_launch:
            sol.persistent(False)
        shape = sol.solve_launch()
        blocks = {SMALL: min(148, -(-sc.fluid_count // 32)), DEEP: 148, WIDE: 296}[form]
        assert shape == {"form": form, "blocks": blocks, "threads": threads}
        a, b = sc.model.state(), sc.model.state()
        l0 = sol.kernel_launches()
        sol.step(a, b, None, None, sc.dt)
        launches.append(sol.kernel_launches() - l0)
    assert launches[0] < launches[1], launches
