"""A hinge that names a vertex twice: two faces on the same three vertices share
all their edges, and each edge's hinge has the third vertex as both of its wings
(what the mesh builder makes of a two-sided triangle).

Tolerance of the blocks: the same expressions in FP64 in another order, 1e-9 of
the largest entry (as for the other terms; the energies and gradients are sums of
a few terms of that size). Tolerance of the steps: the solve moves one corner of a
hinge at a time, the oracle both, so their Newton steps differ and only what the
iteration converges to is common; a vertex whose solve fails stays where it was,
100 % of its way off, and 1 % of the way leaves two orders of magnitude."""
import numpy as np
import pytest

import oracle
from clothcraft_b200 import scenes
from clothcraft_b200.vbd import VbdSolver

pytestmark = pytest.mark.gpu


def two_sided(material, seed, turn, sheet):
    """A triangle with both its faces (turn: the rotation of its vertices' numbers), deformed and moving; with
    `sheet`, beside a 6 x 5 grid whose neighbour lists come before the triangle's and after it."""
    rng = np.random.default_rng(seed)
    uv = np.array([[0.0, 0.0], [0.1, 0.01], [0.03, 0.09]])
    tri = (np.array([[0, 1, 2], [0, 2, 1]]) + turn) % 3
    meshes = [scenes.build_mesh(uv, tri.astype(np.uint32), material)]
    xs = [np.stack([uv[:, 0], np.full(3, 0.5), uv[:, 1]], axis=1)]
    if sheet:
        g = scenes.grid_uv(6, 5, 0.1, 0.08)
        part = scenes.build_mesh(g, scenes.grid_triangles(6, 5, alternate=True), material)
        for side in (0, 2):
            meshes.insert(side, part)
            xs.insert(side, np.stack([g[:, 0], np.full(30, 0.2 + 0.3 * side), g[:, 1]], axis=1))
    x = np.concatenate(xs)
    x = x + rng.uniform(-0.002, 0.002, x.shape)
    v = rng.uniform(-0.02, 0.02, x.shape)
    return scenes.Scene("two-sided", scenes.concat_meshes(meshes), None, x, v,
                        scenes.StepSettings(dt=1 / 60, radius=0.001, stiffness=1e4), 1)


@pytest.mark.parametrize("material", [scenes.Material(), scenes.Material.stvk_mapped()])
@pytest.mark.parametrize("turn,sheet", [(0, False), (1, False), (2, True)])
def test_two_faces_on_three_vertices(material, turn, sheet):
    sc = two_sided(material, 5 + turn, turn, sheet)
    assert any(len(set(h)) == 3 for h in sc.mesh.hinges.tolist())
    st = sc.settings.to_c()
    eg, gg, _ = VbdSolver(sc).local_blocks(sc.x0, 0.002, st)
    eo, go, _ = oracle.Solver(sc).local_blocks(sc.x0, 0.002, st)
    assert np.all(np.abs(eg - eo) <= 1e-9 * np.abs(eo).max())
    assert np.all(np.abs(gg - go) <= 1e-9 * np.abs(go).max())
    for lanes in (1, 4, 8, 32):
        g, o = VbdSolver(sc).set_lanes(lanes), oracle.Solver(sc)
        x, v, t = sc.x0, sc.v0, 0.0
        xo, vo, to = sc.x0, sc.v0, 0.0
        for _ in range(3):
            x, v, t, m = g.step(x, v, t, st)
            xo, vo, to, mo = o.step(xo, vo, to, st)
        way = np.linalg.norm(xo - sc.x0, axis=1)
        assert way.min() > 1e-3 and np.isfinite(m["residual_rms_n"])
        assert np.all(np.linalg.norm(x - xo, axis=1) <= 0.01 * way)
