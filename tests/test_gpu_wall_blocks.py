# SPDX-License-Identifier: Apache-2.0
"""The wall slots' two block shapes (64 particles a block in small models, 256 above two blocks per SM): a world's slots
are the same bits alone and as one of many, particle by particle, near flat walls, in corners and in a bowl."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from alloy_b200.solvers.sph import SolverDFSPH
from alloy_b200.solvers.sph.build import add_fluid_block, add_fluid_points, add_particle_box, add_wall_particles
from alloy_b200.solvers.sph.model import ModelBuilder
from alloy_b200.solvers.sph.testing import benchmark_config, bowl_interior_points, hemisphere_shell_points

pytestmark = pytest.mark.gpu
FIELDS = ("slot_psi", "slot_phi", "slot_g", "slot_vb", "slot_n")


def _fields(cuda, kind, worlds):
    cfg = benchmark_config(0.01)
    b = ModelBuilder(gravity=(0.0, 0.0, -9.81))
    for _ in range(worlds):
        b.begin_world()
        if kind == "box":
            add_fluid_block(b, cfg, (0.0, 0.0, 0.0), (13, 7, 9), jitter=0.02, seed=3)
            add_particle_box(b, cfg, (0.0, 0.0, 0.0), (0.13, 0.07, 0.12), open_top=True)
        else:
            add_fluid_points(b, cfg, bowl_interior_points((0.0, 0.0, 0.08), 0.08, cfg.spacing))
            add_wall_particles(b, cfg, hemisphere_shell_points((0.0, 0.0, 0.08), 0.08, cfg.spacing),
                               velocity=(0.2, -0.1, 0.0))
        b.end_world()
    m = b.finalize(cuda)
    sol = SolverDFSPH(m, cfg)
    s = m.state()
    sol.density_ratio(s)
    torch.cuda.synchronize()
    n = m.particle_count // worlds
    return [sol.debug_field(f).reshape(worlds, n, -1) for f in FIELDS], n


@pytest.mark.parametrize("kind", ["box", "bowl"])
def test_wall_slots_do_not_depend_on_the_block_shape(cuda, kind):
    alone, n = _fields(cuda, kind, 1)
    worlds = 2 * 148 * 256 // n + 2  # past two blocks of 256 per SM
    many, _ = _fields(cuda, kind, worlds)
    assert (alone[0] > 0.0).sum() > 50  # particles with a slot
    has = alone[0][0, :, 0] >= 0.0  # the other fields of an empty slot hold nothing
    np.testing.assert_array_equal(many[0], np.broadcast_to(alone[0], many[0].shape), err_msg=FIELDS[0])
    for name, x, y in zip(FIELDS[1:], alone[1:], many[1:]):
        np.testing.assert_array_equal(y[:, has], np.broadcast_to(x, y.shape)[:, has], err_msg=name)
