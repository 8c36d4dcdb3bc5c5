"""Every register budget and group width of the FP64 sweep against the oracle: the
sweeps at 80 and 64 registers read a solve's records and positions as they need
them, the others ahead, and staged positions end at 4 to 24 neighbours by width.
The scenes have vertices on both sides of that (a grid's 6 to 12, a disc's hub of
41, a border of 5) and contacts of several layers.

Tolerance: one step, 1e-9 m as in the other one-step comparisons with the oracle."""
import numpy as np
import pytest

import oracle
from clothcraft_b200 import scenes
from clothcraft_b200.vbd import VbdSolver

pytestmark = pytest.mark.gpu


def disc_scene():
    a = 2.0 * np.pi * np.arange(41) / 41
    uv = np.concatenate([[[0.0, 0.0]], 0.1 * np.stack([np.cos(a), np.sin(a)], axis=1)])
    i = np.arange(41)
    tri = np.stack([np.zeros(41, int), 1 + i, 1 + (i + 1) % 41], axis=1)
    mesh = scenes.build_mesh(uv, tri.astype(np.uint32), scenes.Material())
    x = np.stack([uv[:, 0], 0.2 + 0.004 * np.sin(3.0 * np.arctan2(uv[:, 1], uv[:, 0])), uv[:, 1]], axis=1)
    x += np.random.default_rng(1).uniform(-2e-4, 2e-4, x.shape)
    return scenes.Scene("disc", mesh, None, x, np.zeros_like(x),
                        scenes.StepSettings(dt=1 / 60, radius=0.001, stiffness=1e4), 1)


def layers_scene():
    rng = np.random.default_rng(2)
    uv = scenes.grid_uv(9, 8, 0.032, 0.028)
    part = scenes.build_mesh(uv, scenes.grid_triangles(9, 8, alternate=True), scenes.Material.stvk_mapped())
    x = np.concatenate([np.stack([uv[:, 0] + 0.0011 * k, np.full(72, 8e-4 * k), uv[:, 1]], axis=1) for k in range(3)])
    x = x + rng.uniform(-5e-5, 5e-5, x.shape)
    return scenes.Scene("layers", scenes.concat_meshes([part] * 3), None, x, np.zeros_like(x),
                        scenes.StepSettings(dt=1 / 60, radius=0.001, stiffness=1e4), 1)


@pytest.mark.parametrize("scene", [disc_scene, layers_scene])
def test_every_width_and_register_budget(scene):
    sc = scene()
    st = sc.settings.to_c()
    x, v, t, m = oracle.Solver(sc, threads=4).step(sc.x0, sc.v0, 0.0, st)
    assert np.abs(x - sc.x0).max() > 1e-4
    wide = [lanes | cap << 8 | 2 << 17 for lanes in (4, 8) for cap in (4, 6, 8)]
    for variant in [lanes | cap << 8 for lanes in (1, 2, 4, 8, 16, 32) for cap in (3, 4, 5, 6, 8)] + wide:
        xg, vg, tg, mg = VbdSolver(sc).set_lanes(variant).step(sc.x0, sc.v0, 0.0, st)
        assert np.abs(xg - x).max() <= 1e-9, hex(variant)
        assert mg["contact_terms"] == m["contact_terms"] and mg["truncated_vertices"] == m["truncated_vertices"]
