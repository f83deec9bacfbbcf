# SPDX-License-Identifier: Apache-2.0
"""A barrier wait of a one-launch solve that gives up: in every form, with either solver, in one world and several, the
kernel ends, the report fails and says what failed, the next step, density field and priming are refused until the status
is cleared, and afterwards the solver steps on as a fresh one does. (Each barrier is told to wait for one block more than
the grid has, with a short limit, so every wait runs out; nothing else is wrong with the launch.)"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from alloy_b200.solvers.sph import SolverDFSPH
from alloy_b200.solvers.sph.testing import dam_break, water_column

pytestmark = pytest.mark.gpu


def _scene(cuda, counts, worlds, solver):
    if worlds > 1:
        return water_column(*counts, worlds=worlds, r=2.0e-3, device=cuda, pressure_solver=solver)
    box = tuple(0.01 * (c + 12) for c in counts)
    return dam_break(counts=counts, box=box, spacing=0.01, dt=5.0e-4, device=cuda, pressure_solver=solver)


def _solver(sc, graphs=True):
    sol = SolverDFSPH(sc.model, sc.config)
    sol.autotune(False)
    sol.use_graphs(graphs)
    return sol


CASES = [
    ((8, 8, 10), 1, "jacobi"),     # rows in shared memory, the step after its rows in one launch
    ((8, 8, 10), 1, "cg"),
    ((8, 8, 10), 3, "jacobi"),
    ((8, 8, 10), 3, "cg"),
    ((36, 36, 36), 1, "jacobi"),   # 46,656 particles: deep blocks
    ((36, 36, 36), 1, "cg"),
    ((16, 16, 16), 12, "jacobi"),  # 49,152 in several worlds
    ((16, 16, 16), 12, "cg"),
    ((54, 54, 54), 1, "jacobi"),   # 157,464: wide blocks
    ((16, 16, 16), 39, "cg"),      # 159,744 in several worlds
]


@pytest.mark.parametrize("counts,worlds,solver", CASES)
def test_the_report_fails_and_the_solver_recovers(cuda, counts, worlds, solver):
    sc, sr = _scene(cuda, counts, worlds, solver), _scene(cuda, counts, worlds, solver)
    sol, ref = _solver(sc), _solver(sr)
    a, b = sc.model.state(), sc.model.state()
    c, d = sr.model.state(), sr.model.state()
    sol.barrier_wait(polls=2000, extra_arrivals=1)
    sol.step(a, b, None, None, sc.dt)
    with pytest.raises(RuntimeError, match="grid-barrier wait"):
        sol.report()
    sol.clear_status()
    sol.barrier_wait()
    a, b = sc.model.state(), sc.model.state()
    mine, theirs = sol.alloy_state_arrays(), ref.alloy_state_arrays()
    for key in ("sph.kappa_v", "sph.kappa_d", "sph.phase", "particle_flags"):
        mine[key].copy_(theirs[key])
    for _ in range(3):
        sol.step(a, b, None, None, sc.dt)
        ref.step(c, d, None, None, sr.dt)
        a, b, c, d = b, a, d, c
    np.testing.assert_array_equal(a.particle_q.cpu().numpy(), c.particle_q.cpu().numpy())
    np.testing.assert_array_equal(a.particle_qd.cpu().numpy(), c.particle_qd.cpu().numpy())
    np.testing.assert_array_equal(sol.report().iters_density, ref.report().iters_density)


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("counts,worlds,solver", [CASES[0], CASES[4]])
def test_the_next_calls_are_refused(cuda, counts, worlds, solver, graphs):
    """Without a report in between: once the failed launch has ended, the calls that would go on from its results say so."""
    sc = _scene(cuda, counts, worlds, solver)
    sol = _solver(sc, graphs)
    a, b = sc.model.state(), sc.model.state()
    sol.barrier_wait(polls=2000, extra_arrivals=1)
    sol.step(a, b, None, None, sc.dt)
    torch.cuda.synchronize()
    for call in (lambda: sol.step(b, a, None, None, sc.dt), lambda: sol.density_ratio(b), lambda: sol.prime(b, sc.dt),
                 sol.report):
        with pytest.raises(RuntimeError, match="grid-barrier wait"):
            call()
    sol.clear_status()
    sol.barrier_wait()
    a = sc.model.state()
    sol.density_ratio(a)
    sol.prime(a, sc.dt)
    sol.step(a, b, None, None, sc.dt)
    sol.report()


def test_a_priming_that_fails_says_so(cuda):
    sc = _scene(cuda, (8, 8, 10), 2, "cg")
    sol = _solver(sc)
    sol.barrier_wait(polls=2000, extra_arrivals=1)
    with pytest.raises(RuntimeError, match="grid-barrier wait"):
        sol.prime(sc.model.state(), sc.dt)
    sol.clear_status()
    sol.barrier_wait()
    sol.prime(sc.model.state(), sc.dt)
    sol.report()


@pytest.mark.parametrize("solver", ["jacobi", "cg"])
def test_the_message_names_the_launch_that_failed(cuda, solver):
    sc = _scene(cuda, (8, 8, 10), 1, solver)
    sol = _solver(sc)
    a, b = sc.model.state(), sc.model.state()
    sol.barrier_wait(polls=2000, extra_arrivals=1)
    sol.step(a, b, None, None, sc.dt)
    with pytest.raises(RuntimeError, match="grid-barrier wait of a solve in one launch"):
        sol.report()
