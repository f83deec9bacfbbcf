# SPDX-License-Identifier: Apache-2.0
"""Whole pressure solves as one cooperative launch against one kernel per phase (the path the oracle's tests pin), bit for
bit: a lone particle, rows and blocks that end raggedly, the sizes on both sides of each form's limit (rows in shared
memory up to 256 particles per SM; deep blocks; wide ones where they save a round), one world and several, Jacobi and CG,
particle and shape walls, rows longer than the resident ones, and liquid that outgrew the shape chosen at creation."""

from __future__ import annotations

import numpy as np
import pytest

from alloy_b200.solvers.sph import SolverDFSPH
from alloy_b200.solvers.sph.build import add_box_tank, add_fluid_block, add_particle_box
from alloy_b200.solvers.sph.model import ModelBuilder, ParticleFlags
from alloy_b200.solvers.sph.testing import benchmark_config

pytestmark = pytest.mark.gpu
DT = 5.0e-4


def _model(device, counts, worlds, walls, cfg, squeeze=1.0, asleep=0):
    s = cfg.spacing
    b = ModelBuilder(gravity=(0.0, 0.0, -9.81))
    for w in range(worlds):
        b.begin_world()
        # uneven worlds: the last axis differs
        nz = max(counts[2] - w % 3, 1)
        add_fluid_block(b, cfg, (0.0, 0.0, 0.0), (counts[0], counts[1], nz), jitter=0.02, seed=w, velocity=(0.3, 0.1, 0.0))
        box = tuple(float((c + 4) * s) for c in (counts[0], counts[1], counts[2]))
        if walls == "sdf":
            add_box_tank(b, (0.0, 0.0, 0.0), box, wall=cfg.h)
        else:
            add_particle_box(b, cfg, (0.0, 0.0, 0.0), box, open_top=True)
        if asleep:
            x = np.stack(np.meshgrid(*[np.arange(8)] * 3, indexing="ij"), -1).reshape(-1, 3)[:asleep]
            b.add_particles((x + 0.5) * s, (0.0, 0.0, 0.0), 1000.0 * s**3, cfg.particle_radius, int(ParticleFlags.ACTIVE),
                            -1, 1000.0)
        b.end_world()
    m = b.finalize(device)
    m.particle_q.mul_(squeeze)
    return m


def _same(cuda, make, steps, wake=None):
    runs = []
    for one_launch in (True, False):
        model, cfg = make()
        sol = SolverDFSPH(model, cfg)
        sol.autotune(False)
        if not one_launch:
            sol.persistent(False)
        if wake is not None:
            wake(model)
        a, b = model.state(), model.state()
        its = []
        for _ in range(steps):
            sol.step(a, b, None, None, DT)
            a, b = b, a
            r = sol.report()  # raises if a barrier wait gave up
            its.append(np.concatenate([r.iters_density, r.iters_divergence, r.density_err, r.divergence_err]))
        k = sol.alloy_state_arrays()
        runs.append([t.cpu().numpy() for t in (a.particle_q, a.particle_qd, k["sph.kappa_v"], k["sph.kappa_d"])] +
                    [np.stack(its)])
    for name, x, y in zip(("q", "qd", "kappa_v", "kappa_d", "statistics"), *runs):
        np.testing.assert_array_equal(x, y, err_msg=name)
    return runs[0]


@pytest.mark.parametrize("counts,worlds,walls,solver,steps", [
    ((1, 1, 1), 1, "particles", "jacobi", 3),        # one particle, no neighbour
    ((5, 7, 1), 1, "sdf", "cg", 3),                  # one block, its second warp almost empty
    ((5, 7, 3), 5, "particles", "cg", 6),            # several tiny worlds
    ((33, 33, 34), 1, "particles", "jacobi", 3),     # 37,026: rows in shared memory, blocks almost full
    ((33, 34, 34), 1, "sdf", "cg", 3),               # 38,148: just past them
    ((23, 22, 25), 3, "particles", "jacobi", 3),     # 36,432 in three worlds
    ((23, 25, 25), 3, "sdf", "cg", 3),               # 41,400 in three worlds
    ((54, 54, 54), 1, "sdf", "jacobi", 2),           # 157,464: wide blocks
    ((17, 16, 16), 39, "particles", "cg", 2),        # 159,120 in 39 worlds: wide blocks
])
def test_one_launch_equals_one_kernel_per_phase(cuda, counts, worlds, walls, solver, steps):
    cfg = benchmark_config(0.01, pressure_solver=solver)
    _same(cuda, lambda: (_model(cuda, counts, worlds, walls, cfg), cfg), steps)


@pytest.mark.parametrize("solver", ["jacobi", "cg"])
def test_rows_longer_than_the_resident_ones(cuda, solver):
    cfg = benchmark_config(0.01, pressure_solver=solver)
    make = lambda: (_model(cuda, (10, 9, 11), 1, "particles", cfg, squeeze=0.82), cfg)  # noqa: E731
    model, _ = make()
    sol = SolverDFSPH(model, cfg)
    a, b = model.state(), model.state()
    sol.step(a, b, None, None, DT)
    assert sol.neighbor_rows()[1].max() > 40
    _same(cuda, make, 2)


@pytest.mark.parametrize("solver", ["jacobi", "cg"])
def test_liquid_that_outgrew_the_launch(cuda, solver):
    """Particles outside the solver's groups at creation become liquid afterwards: more than the blocks hold."""
    cfg = benchmark_config(0.01, pressure_solver=solver)

    def wake(model):
        ph = model.sph.phase
        ph[(model.particle_flags == int(ParticleFlags.ACTIVE)) & (ph == -1)] = 1

    out = _same(cuda, lambda: (_model(cuda, (3, 3, 2), 1, "sdf", cfg, asleep=400), cfg), 3, wake)
    assert np.abs(out[1]).max() > 0.0
