"""The colouring walk against the oracle's sequential greedy where it takes its
different routes: rows with several neighbours of the same chunk and warp,
vertex orders in which neighbours lie far apart, rows that overflow and more
than 64 colours (the full rule), and sizes around a warp and a chunk."""
import numpy as np
import pytest

import oracle
from clothcraft_b200 import scenes
from clothcraft_b200.vbd import VbdSolver

pytestmark = pytest.mark.gpu


def layers(nx, ny, count, gap, permute=None, seed=0):
    """`count` grids of nx x ny vertices, 4 mm apart, stacked `gap` metres apart."""
    rng = np.random.default_rng(seed)
    uv = scenes.grid_uv(nx, ny, 0.004 * (nx - 1), 0.004 * (ny - 1))
    n = len(uv)
    tri = np.concatenate([scenes.grid_triangles(nx, ny, alternate=False).astype(np.int64) + k * n for k in range(count)])
    x = np.concatenate([np.stack([uv[:, 0] + 0.0011 * k % 0.004, np.full(n, gap * k), uv[:, 1] + 0.0007 * k % 0.004], axis=1)
                        for k in range(count)])
    x = x + rng.uniform(-0.1 * gap, 0.1 * gap, x.shape)
    uv = np.concatenate([uv + [0.0, 0.05 * (ny + 1) * k] for k in range(count)])
    order = np.arange(len(x))
    if permute == "random":
        order = rng.permutation(len(x))
    elif permute == "interleaved":  # the layers' vertices in turn: a stack's column is one warp
        order = order.reshape(count, n).T.ravel()
    inverse = np.empty_like(order)
    inverse[order] = np.arange(len(order))
    mesh = scenes.build_mesh(uv[order], inverse[tri].astype(np.uint32), scenes.Material.stvk_mapped())
    s = scenes.StepSettings(dt=1 / 60, radius=0.001, stiffness=1e4)
    return scenes.Scene("layers", mesh, None, np.ascontiguousarray(x[order]), np.zeros_like(x), s, 1)


@pytest.mark.parametrize("nx,ny,count,gap,rq,permute,least", [
    (3, 2, 1, 1e-3, 4e-3, None, 4),               # fewer vertices than a warp
    (31, 33, 1, 1e-3, 4e-3, None, 4),             # one vertex short of a chunk
    (32, 32, 1, 1e-3, 4e-3, None, 4),             # a chunk
    (41, 25, 2, 1e-3, 4e-3, None, 5),             # a chunk and one vertex, two layers
    (41, 25, 2, 1e-3, 4e-3, "random", 5),         # neighbours in other chunks
    (23, 17, 6, 5e-4, 4e-3, "interleaved", 6),    # contacts within a warp
    (60, 30, 5, 5e-4, 4e-3, None, 6),             # contacts 1-4 chunks away
    (12, 11, 48, 1e-4, 4e-3, None, 65),           # more than 64 colours, rows of more than 64 neighbours
    (12, 11, 48, 1e-4, 4e-3, "interleaved", 65),
    (12, 11, 48, 1e-4, 4e-3, "random", 65),
])
def test_walk_equals_sequential_greedy(nx, ny, count, gap, rq, permute, least):
    sc = layers(nx, ny, count, gap, permute)
    g = VbdSolver(sc)
    o = oracle.Solver(sc, threads=8)
    n = sc.n
    grab = dict(vertices=[n - 1, n // 2, 0], weights=[0.2, 0.3, 0.5], target=[0.0, 0.2, 0.0], stiffness=100.0)
    for k, gr in enumerate((None, grab, None)):  # from scratch, from the last colouring, and after a displacement
        x = sc.x0.copy()
        if k == 2:
            x[::5, 1] += 0.2 * gap
        cg, ng = g.colors(x, rq, sc.settings, grab=gr)
        co, no = o.colors(x, rq, sc.settings.ogc_c(), grab=gr)
        assert ng == no and ng >= least
        assert np.array_equal(cg, co)


@pytest.mark.parametrize("nx,ny", [(2, 2), (33, 32), (33, 33), (2, 1026), (41, 50), (32, 64), (3, 683)])
def test_small_sorts_around_their_limit(nx, ny):
    """Triangle counts 2, 1984, 2048 and 2050 (the extension metric's sort), vertex counts 2050, 2048 and 2049 (the
    colour order): a step takes every vertex in its colour's turn and reports the metric of the sorted strains."""
    sc = layers(nx, ny, 1, 1e-3, "random", seed=nx)
    st = sc.settings.to_c()
    x, v, t, m = VbdSolver(sc).step(sc.x0, sc.v0, 0.0, st)
    xo, vo, to, mo = oracle.Solver(sc, threads=8).step(sc.x0, sc.v0, 0.0, st)
    # positions as in the other one-step comparisons; the metric moves with them by 100 / (4 mm spacing) per metre
    assert np.abs(x - xo).max() <= 1e-9
    assert abs(m["extension_p95_percent"] - mo["extension_p95_percent"]) <= 1e-4
    assert abs(m["extension_max_percent"] - mo["extension_max_percent"]) <= 1e-4
    assert m["extension_max_percent"] >= m["extension_p95_percent"] > 0.0
