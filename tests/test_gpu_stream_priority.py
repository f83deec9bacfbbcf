# SPDX-License-Identifier: Apache-2.0
"""Steps on streams of raised priority run one kernel per phase, at the stream's own priority: a solve as one launch holds
every SM until its last barrier, and two such launches of different priorities could each hold part of the SMs. Solvers
stepping at once from two threads, on streams of equal and of different priorities, compute what each computes alone."""

from __future__ import annotations

import threading

import numpy as np
import pytest
import torch

from alloy_b200.solvers.sph import SolverDFSPH
from alloy_b200.solvers.sph.testing import dam_break, water_column

pytestmark = pytest.mark.gpu


def _scene(cuda, kind):
    if kind == "columns":
        return water_column(12, 12, 12, worlds=2, r=2.0e-3, device=cuda)
    return dam_break(counts=(40, 33, 31), box=(0.9, 0.6, 0.6), spacing=0.01, dt=5.0e-4, device=cuda)


def _steps(cuda, kind, stream, steps=12, graphs=True, per_phase=False):
    with torch.cuda.stream(stream):
        sc = _scene(cuda, kind)
        sol = SolverDFSPH(sc.model, sc.config)
        sol.autotune(False)
        sol.use_graphs(graphs)
        if per_phase:
            sol.persistent(False)
        a, b = sc.model.state(), sc.model.state()
        l0 = sol.kernel_launches()
        for _ in range(steps):
            sol.step(a, b, None, None, sc.dt)
            a, b = b, a
        stream.synchronize()  # the iterations inside replayed graphs are counted on the device
        launches = sol.kernel_launches() - l0
        sol.report()  # raises if a barrier wait gave up
        return a.particle_q.cpu().numpy(), a.particle_qd.cpu().numpy(), launches


@pytest.mark.parametrize("kind", ["columns", "dam"])
@pytest.mark.parametrize("graphs", [True, False])
def test_raised_priority_takes_one_kernel_per_phase(cuda, kind, graphs):
    ordinary = _steps(cuda, kind, torch.cuda.Stream(priority=0), graphs=graphs)
    raised = _steps(cuda, kind, torch.cuda.Stream(priority=-1), graphs=graphs)
    phases = _steps(cuda, kind, torch.cuda.Stream(priority=0), graphs=graphs, per_phase=True)
    assert raised[2] == phases[2] and raised[2] != ordinary[2], (ordinary[2], raised[2], phases[2])
    for x, y in zip(ordinary[:2], raised[:2]):
        np.testing.assert_array_equal(x, y)


def test_one_solver_on_streams_of_both_kinds(cuda):
    """The form follows the stream of each step, replayed graphs included."""
    sc = _scene(cuda, "dam")
    sol = SolverDFSPH(sc.model, sc.config)
    sol.autotune(False)
    a, b = sc.model.state(), sc.model.state()
    streams = [torch.cuda.Stream(priority=0), torch.cuda.Stream(priority=-1)]
    torch.cuda.synchronize()
    counts = [[], []]
    for k in range(8):
        i = (k // 2) % 2  # two steps on each, so that both state orders' graphs are replayed on both streams
        with torch.cuda.stream(streams[i]):
            l0 = sol.kernel_launches()
            sol.step(a, b, None, None, sc.dt)
            streams[i].synchronize()
            counts[i].append(sol.kernel_launches() - l0)
            a, b = b, a
    assert min(counts[1]) > max(counts[0]) == min(counts[0]), counts
    np.testing.assert_array_equal(a.particle_q.cpu().numpy(),
                                  _steps(cuda, "dam", torch.cuda.Stream(priority=0), steps=8)[0])


@pytest.mark.parametrize("priorities", [(0, 0), (-1, 0), (0, -1), (-1, -2)])
def test_two_solvers_at_once(cuda, priorities):
    kinds = ("columns", "dam")
    alone = [_steps(cuda, k, torch.cuda.Stream(priority=0), steps=40) for k in kinds]
    both, errors = [None, None], []

    def work(i):
        try:
            both[i] = _steps(cuda, kinds[i], torch.cuda.Stream(priority=priorities[i]), steps=40)
        except Exception as e:  # shown by the assertion below
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for x, y in zip(alone, both):
        np.testing.assert_array_equal(x[0], y[0])
        np.testing.assert_array_equal(x[1], y[1])
