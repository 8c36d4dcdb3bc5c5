"""The colouring walk against the oracle's sequential greedy for hubs (vertices with
hundreds or thousands of neighbours, more than a row holds) and for changes far
apart in the vertex order (most chunks left out, also beyond one scan of 32)."""
import numpy as np
import pytest

import oracle
from clothcraft_b200 import scenes
from clothcraft_b200.vbd import VbdSolver

pytestmark = pytest.mark.gpu


def disc(rim, hub):
    """A fan of triangles around one vertex, numbered `hub`."""
    a = 2.0 * np.pi * np.arange(rim) / rim
    uv = 0.3 * np.stack([np.cos(a), np.sin(a)], axis=1)
    uv = np.insert(uv, hub, [0.0, 0.0], axis=0)
    around = np.delete(np.arange(rim + 1), hub)
    tri = np.stack([np.full(rim, hub), around, np.roll(around, -1)], axis=1)
    mesh = scenes.build_mesh(uv, tri.astype(np.uint32), scenes.Material.stvk_mapped())
    x = np.stack([uv[:, 0], 0.01 * np.sin(40.0 * uv[:, 0]), uv[:, 1]], axis=1)
    s = scenes.StepSettings(dt=1 / 60, radius=0.25 * np.pi * 0.3 / rim, stiffness=1e4)
    return scenes.Scene("disc", mesh, None, x, np.zeros_like(x), s, 1)


@pytest.mark.parametrize("rim,hub", [(60, 60), (70, 70), (300, 0), (300, 150), (300, 300), (2500, 2500), (2500, 1024)])
def test_hub_colours_equal_sequential_greedy(rim, hub):
    sc = disc(rim, hub)
    g, o = VbdSolver(sc), oracle.Solver(sc, threads=4)
    grab = dict(vertices=[rim, rim // 2, 1], weights=[0.2, 0.3, 0.5], target=[0.0, 0.2, 0.0], stiffness=100.0)
    for gr in (None, grab, None):
        cg, ng = g.colors(sc.x0, 3 * sc.settings.radius, sc.settings, grab=gr)
        co, no = o.colors(sc.x0, 3 * sc.settings.radius, sc.settings.ogc_c(), grab=gr)
        assert ng == no and np.array_equal(cg, co)


@pytest.mark.parametrize("count", [565, 903, 1600])
def test_sparse_changes_equal_sequential_greedy(count):
    """Separate 8 x 8 patches, 36,160 and 57,792 vertices (colours in shared memory; two scans) and 102,400 (colours in
    global memory, four). A grab of three vertices of one colour in patches far apart makes two of them change, and at
    most their patches with them; letting go changes them back."""
    uv = scenes.grid_uv(8, 8, 0.028, 0.028)
    k = np.repeat(np.arange(count), 64)[:, None]
    uv = np.tile(uv, (count, 1)) + 0.05 * np.concatenate([k % 40, k // 40], axis=1)
    tri = scenes.grid_triangles(8, 8, alternate=False).astype(np.int64)
    tri = (tri[None] + 64 * np.arange(count)[:, None, None]).reshape(-1, 3)
    mesh = scenes.build_mesh(uv, tri.astype(np.uint32), scenes.Material.stvk_mapped())
    x = np.stack([uv[:, 0], np.zeros(len(uv)), uv[:, 1]], axis=1)
    sc = scenes.Scene("patches", mesh, None, x, np.zeros_like(x), scenes.StepSettings(dt=1 / 60, radius=5e-4, stiffness=1e4), 1)
    g, o = VbdSolver(sc), oracle.Solver(sc, threads=8)
    n = sc.n
    first, _ = g.colors(x, 0.002, sc.settings)
    same = np.flatnonzero(first == first[5])
    ends = [same[same > 40][0], same[-2]]
    middle = same[len(same) // 2]
    early = same[same > 1024][0]
    for vertices in (None, [ends[0], middle, ends[1]], None, [ends[0], early, ends[1]], [early, middle, ends[1]], None):
        gr = None
        if vertices is not None:
            gr = dict(vertices=[int(v) for v in vertices], weights=[0.2, 0.3, 0.5], target=[0.0, 0.2, 0.0], stiffness=100.0)
        cg, ng = g.colors(x, 0.002, sc.settings, grab=gr)
        co, no = o.colors(x, 0.002, sc.settings.ogc_c(), grab=gr)
        assert ng == no and np.array_equal(cg, co)
        if vertices is not None:
            assert 0 < np.count_nonzero(cg != first) <= 3 * 64
