# SPDX-License-Identifier: Apache-2.0
"""One kernel per phase, asked for with persistent(False): what Jacobi models of many millions of particles, solvers with
item halos and streams of raised priority run, while an ordinary step runs each solve as one launch. The tuner's choices
and every pinned choice give the same bits in graph-replayed steps; the Jacobi and both forms of the CG products equal the
oracle's restatement bit for bit."""

from __future__ import annotations

import numpy as np
import pytest

from alloy_b200 import _lib
from alloy_b200.solvers.sph import SolverDFSPH
from alloy_b200.solvers.sph.testing import batched_worlds, dam_break
from oracle.pyoracle import Oracle

pytestmark = pytest.mark.gpu


def _steps(cuda, tune=False, pins=()):
    sc = batched_worlds(worlds=4, lo=1500, hi=6000, seed=5, device=cuda)
    sol = SolverDFSPH(sc.model, sc.config)
    sol.persistent(False)
    sol.autotune(tune)
    for name, block, nb in pins:
        sol.set_tuned_config(name, block, nb)
    a, b = sc.model.state(), sc.model.state()
    for _ in range(6):
        sol.step(a, b, None, None, sc.dt)
        a, b = b, a
    r = sol.report()
    return [a.particle_q.cpu().numpy(), a.particle_qd.cpu().numpy(), r.iters_density, r.iters_divergence, r.density_err]


def test_every_configuration_gives_the_same_bits(cuda):
    want = _steps(cuda)
    names = [k for k in _lib.TUNE_KERNELS if k != "lists"]
    runs = [_steps(cuda, tune=True)]
    runs += [_steps(cuda, pins=[(k, block, nb) for k in names]) for block in (128, 256) for nb in (4, 8, 16)]
    for got in runs:
        for x, y in zip(want, got):
            np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("counts,solver,steps", [
    ((12, 10, 14), "jacobi", 12),
    ((12, 10, 14), "cg", 12),   # the CG products by teams of four lanes
    ((56, 48, 52), "cg", 3),    # more than 131,072 particles: one lane per particle
])
def test_equals_the_oracle(cuda, counts, solver, steps):
    sc = dam_break(counts=counts, box=(0.8, 0.6, 0.8), spacing=0.01, device=cuda, pressure_solver=solver)
    sol = SolverDFSPH(sc.model, sc.config)
    sol.persistent(False)
    orc = Oracle(sc.model.host(), sc.config)
    a, b = sc.model.state(), sc.model.state()
    for k in range(steps):
        sol.step(a, b, None, None, sc.dt)
        a, b = b, a
        orc.step(sc.dt)
        q, qd = orc.state()
        np.testing.assert_array_equal(a.particle_q.cpu().numpy(), q, err_msg=f"q step {k}")
        np.testing.assert_array_equal(a.particle_qd.cpu().numpy(), qd, err_msg=f"qd step {k}")
        rep, orep = sol.report(), orc.report()
        np.testing.assert_array_equal(rep.iters_density, orep["iters_density"], err_msg=f"step {k}")
        np.testing.assert_array_equal(rep.iters_divergence, orep["iters_divergence"], err_msg=f"step {k}")
    kv, kd = orc.warm()
    np.testing.assert_array_equal(sol.alloy_state_arrays()["sph.kappa_v"].cpu().numpy(), kv)
    np.testing.assert_array_equal(sol.alloy_state_arrays()["sph.kappa_d"].cpu().numpy(), kd)
