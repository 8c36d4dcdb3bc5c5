"""Closed-form gradients and Hessians of the local terms against the oracle's
forward differentiation, with every role a vertex can have in a contact and in
a hinge, mollified edge pairs among them.

Tolerance: the oracle and the kernels evaluate the same expressions in FP64 in
another order. A distance of ~1e-3 m between points a metre from the origin
carries 1e-16 / 1e-3 = 1e-13 of relative rounding, and the log barrier's second
derivative k tau^2 / d^2 and the mollifier's 2 / eps raise it by at most a few
hundred: 1e-9 of the block's largest entry leaves an order of magnitude."""
import numpy as np
import pytest

import oracle
from clothcraft_b200 import scenes
from clothcraft_b200.vbd import VbdSolver

pytestmark = pytest.mark.gpu


def two_layers(shift, turn, gap, jitter, material, seed):
    """Two 9 x 8 grids of 4 mm cells, the upper one shifted and turned in its plane."""
    rng = np.random.default_rng(seed)
    meshes, xs = [], []
    for k in range(2):
        uv = scenes.grid_uv(9, 8, 0.032, 0.028)
        meshes.append(scenes.build_mesh(uv, scenes.grid_triangles(9, 8, alternate=True), material))
        c, s = np.cos(turn * k), np.sin(turn * k)
        p = uv @ np.array([[c, s], [-s, c]]) + np.array(shift) * k
        xs.append(np.stack([p[:, 0], np.full(len(p), gap * k), p[:, 1]], axis=1))
    x = np.concatenate(xs) + rng.uniform(-jitter, jitter, (144, 3))
    return scenes.Scene("two", scenes.concat_meshes(meshes), None, x, np.zeros_like(x),
                        scenes.StepSettings(dt=1 / 60, radius=0.002, stiffness=1e4), 1)


@pytest.mark.parametrize("shift,turn,gap,jitter,material", [
    ((0.0011, 0.0007), 0.0, 1.2e-3, 5e-5, scenes.Material.stvk_mapped()),   # parallel edges: mollified pairs
    ((0.0011, 0.0007), 0.4, 1.2e-3, 2e-4, scenes.Material()),               # crossing edges, compression law
    ((0.03, 0.0), 0.1, 0.9e-3, 2e-4, scenes.Material()),                    # layers side by side: borders, points, ends
    ((0.0005, 0.0031), 0.7, 0.7e-3, 2e-4, scenes.Material.stvk_mapped()),   # below half the radius: the log part
])
def test_blocks_match_forward_differentiation(shift, turn, gap, jitter, material):
    roles = set()
    for seed in range(3):
        sc = two_layers(shift, turn, gap, jitter, material, seed)
        g, o = VbdSolver(sc), oracle.Solver(sc)
        st = sc.settings.to_c()
        c = oracle.World(sc.x0, sc.mesh.triangles, sc.n).detect(sc.x0, 0.004, sc.settings.ogc_c())
        roles |= set(np.unique(c["kinds"]).tolist())
        eg, gg, hg = g.local_blocks(sc.x0, 0.004, st)
        eo, go, ho = o.local_blocks(sc.x0, 0.004, st)
        assert np.all(np.abs(eg - eo) <= 1e-9 * np.abs(eo).max())
        assert np.all(np.abs(gg - go) <= 1e-9 * np.maximum(np.linalg.norm(go, axis=1, keepdims=True), np.abs(go).max() * 1e-3))
        assert np.all(np.abs(hg - ho) <= 1e-9 * np.abs(ho).max(axis=(1, 2), keepdims=True))
    assert 3 in roles and 2 in roles
