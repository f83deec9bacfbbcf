# SPDX-License-Identifier: Apache-2.0
"""Whole pressure solves as one cooperative launch against one kernel per phase, bit for bit, where the forms' own
bookkeeping is at work: uneven worlds that stop at different iterations (the lists of the worlds still iterating, the few
runs left that are shared out evenly) on both sides of the limits between the forms, with the Jacobi and the CG, particle
and shape walls; and solves that go on from a judged learned start (the launch's iterations without its start)."""

from __future__ import annotations

import numpy as np
import pytest

from alloy_b200.solvers.sph import SolverDFSPH
from alloy_b200.solvers.sph.build import add_box_tank, add_fluid_block, add_particle_box
from alloy_b200.solvers.sph.model import ModelBuilder
from alloy_b200.solvers.sph.testing import benchmark_config
from alloy_b200.solvers.sph.warmstart import default_model

pytestmark = pytest.mark.gpu
DT = 5.0e-4


def _worlds(device, heights, walls, cfg):
    """One 17 x 16 block per world, of the given number of layers; some are at rest, some fall and are squeezed."""
    s = cfg.spacing
    squeezed = []
    b = ModelBuilder(gravity=(0.0, 0.0, -9.81))
    for w, nz in enumerate(heights):
        b.begin_world()
        v = (0.0, 0.0, -1.0) if w % 4 == 1 else (0.0, 0.0, 0.0)
        ids = add_fluid_block(b, cfg, (0.0, 0.0, 0.0), (17, 16, nz), jitter=0.02, seed=w, velocity=v)
        if w % 4 == 1:
            squeezed.append(ids)
        box = (21 * s, 20 * s, (nz + 4) * s)
        if walls == "sdf":
            add_box_tank(b, (0.0, 0.0, 0.0), box, wall=cfg.h)
        else:
            add_particle_box(b, cfg, (0.0, 0.0, 0.0), box, open_top=True)
        b.end_world()
    m = b.finalize(device)
    for ids in squeezed:
        m.particle_q[ids.start:ids.stop] *= 0.96
    return m


def _heights(layers):
    """Uneven worlds of 3, 8, 15 and 22 layers and a last one that makes up the total."""
    out, left = [], layers
    while left > 30:
        out.append((3, 8, 15, 22)[len(out) % 4])
        left -= out[-1]
    return out + [left]


def _run(cuda, heights, walls, solver, steps, one_launch, learned):
    cfg = benchmark_config(0.01, pressure_solver=solver)
    model = _worlds(cuda, heights, walls, cfg)
    sol = SolverDFSPH(model, cfg)
    sol.autotune(False)
    sol.use_graphs(False)  # eager steps count every launch
    if not one_launch:
        sol.persistent(False)
    if learned:
        sol.set_warm_model(default_model())
    a, b = model.state(), model.state()
    its, kept, l0 = [], 0, sol.kernel_launches()
    for _ in range(steps):
        sol.step(a, b, None, None, DT)
        a, b = b, a
        r = sol.report()  # raises if a barrier wait gave up
        its.append(np.concatenate([r.iters_density, r.iters_divergence, r.density_err, r.divergence_err]))
        if learned:
            d = sol.diagnostics()
            kept += int(d["learned_density"].sum() + d["learned_divergence"].sum())
    launches = sol.kernel_launches() - l0
    k = sol.alloy_state_arrays()
    out = [t.cpu().numpy() for t in (a.particle_q, a.particle_qd, k["sph.kappa_v"], k["sph.kappa_d"])] + [np.stack(its)]
    return out, launches, kept


def _both(cuda, heights, walls, solver, steps, learned=False):
    (one, n_one, kept), (phases, n_phases, _) = [_run(cuda, heights, walls, solver, steps, x, learned)
                                                 for x in (True, False)]
    assert n_one < n_phases, (n_one, n_phases)  # the two runs took different paths
    for name, x, y in zip(("q", "qd", "kappa_v", "kappa_d", "statistics"), one, phases):
        np.testing.assert_array_equal(x, y, err_msg=name)
    if len(heights) > 1:
        its = one[4][:, :len(heights)]
        assert (its.max(axis=1) > its.min(axis=1)).any(), its  # some world stopped before another
    return kept


# 272 particles a layer; on 148 SMs the deep form holds 151,552 particles a round, the wide one 189,440
@pytest.mark.parametrize("layers,walls,solver", [
    (557, "particles", "jacobi"),   # 151,504 particles: deep, one round
    (557, "sdf", "cg"),
    (559, "sdf", "jacobi"),         # 152,048: wide, where the deep form would take a second round
    (559, "particles", "cg"),
    (700, "particles", "jacobi"),   # 190,400: deep, two rounds either way
    (1114, "sdf", "jacobi"),        # 303,008: deep, the second round full
    (1116, "particles", "jacobi"),  # 303,552: wide, two rounds against three
    (140, "sdf", "jacobi"),         # 38,080: deep blocks of 288 threads, the rows just past shared memory
])
def test_uneven_worlds(cuda, layers, walls, solver):
    heights = _heights(layers)
    assert sum(heights) == layers and min(heights) >= 1
    _both(cuda, heights, walls, solver, 3)


@pytest.mark.parametrize("heights,walls,solver", [
    ((150,), "particles", "jacobi"),       # one world, 40,800 particles: deep
    ((170,), "sdf", "cg"),
    (_heights(200), "particles", "jacobi"),  # several worlds, deep
    (_heights(600), "sdf", "jacobi"),        # several worlds, wide
    (_heights(100), "particles", "jacobi"),  # several worlds, rows in shared memory
])
def test_solves_that_go_on_from_a_learned_start(cuda, heights, walls, solver):
    kept = _both(cuda, list(heights), walls, solver, 4, learned=True)
    assert solver == "cg" or kept > 0  # some solve did go on from the network's start
