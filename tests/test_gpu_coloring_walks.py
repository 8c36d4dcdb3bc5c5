"""The colouring walk against the oracle's sequential greedy for hubs: vertices
with hundreds or thousands of neighbours, more than a row holds."""
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
