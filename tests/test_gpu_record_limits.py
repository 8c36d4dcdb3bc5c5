"""Meshes beyond what the sweep's packed records hold: a vertex with more than
2^21 mesh neighbours and a mesh of more than 2^22 materials. Nothing but their
size is special about them."""
import ctypes as C

import numpy as np
import pytest

import oracle
from clothcraft_b200 import abi, scenes
from clothcraft_b200.vbd import VbdSolver

pytestmark = pytest.mark.gpu

PLACES = 1 << 21
MATERIALS = 1 << 22


class ManyMaterials:
    """A mesh whose materials stand at the given numbers of a list of `count`."""

    def __init__(self, mesh, at, count):
        self.mesh, self.at, self.count, self.n = mesh, np.asarray(at, np.uint32), count, mesh.n

    def to_c(self):
        m, keep = self.mesh.to_c()
        fields = len(abi.cc_material._fields_)
        table = np.full((self.count, fields), 7.0)
        table[:, 9] = 0.0
        for k, mat in zip(self.at, self.mesh.materials):
            table[k] = [getattr(mat, name) for name, _ in abi.cc_material._fields_]
        tm, hm = self.at[self.mesh.triangle_material], self.at[self.mesh.hinge_material]
        m.n_materials = self.count
        m.materials = C.cast(table.ctypes.data, C.POINTER(abi.cc_material))
        m.triangle_material = abi.ptr(tm, C.c_uint32)
        m.hinge_material = abi.ptr(hm, C.c_uint32)
        return m, (keep, table, tm, hm)


def test_more_materials_than_a_record_holds():
    """Four materials at numbers on both sides of the limit against the same numbered 0 to 3: one step with residual
    checks, a Newton step and the blocks. The kernels evaluate the same expressions in FP64, rounded differently at most
    where the compiler contracts them: 1e-9 m as in the other one-step comparisons, 1e-9 of the largest entry for the
    blocks and 1e-6 of the residuals (a wrong material's transition moves vertices by 1e-5 m and more)."""
    kinds = [scenes.Material(compression_ratio=0.1 + 0.2 * k, compression_transition=0.003 + 0.004 * k) for k in range(4)]
    uv = scenes.grid_uv(9, 8, 0.2, 0.2)
    mesh = scenes.concat_meshes([scenes.build_mesh(uv, scenes.grid_triangles(9, 8, alternate=True), k) for k in kinds])
    rng = np.random.default_rng(4)
    x = np.concatenate([np.stack([uv[:, 0], np.full(72, 0.1 * k), uv[:, 1]], axis=1) for k in range(4)])
    x = x + rng.uniform(-0.003, 0.003, x.shape)
    few = scenes.Scene("few", mesh, None, x, np.zeros_like(x), scenes.StepSettings(dt=1 / 60, radius=0.001, stiffness=1e4), 1)
    many = scenes.Scene("many", ManyMaterials(mesh, [5, MATERIALS - 2, MATERIALS - 1, MATERIALS + 2], MATERIALS + 3), None, x,
                        np.zeros_like(x), few.settings, 1)
    st = few.settings.to_c()
    st.residual_check_every = 4
    v = np.zeros_like(x)
    a, b = [VbdSolver(sc).set_lanes(8).step(x, v, 0.0, st) for sc in (few, many)]
    assert np.abs(a[0] - b[0]).max() <= 1e-9 and np.abs(a[0] - x).max() > 1e-4
    for key in ("relative_residual", "relative_force_residual", "initial_relative_residual"):
        assert abs(a[3][key] - b[3][key]) <= 1e-6 * a[3][key]
    a, b = [VbdSolver(sc).newton_step(x, v, st)[0] for sc in (few, many)]
    assert np.abs(a - b).max() <= 1e-9
    for p, q in zip(*[VbdSolver(sc).local_blocks(x, 0.002, st) for sc in (few, many)]):
        assert np.abs(p - q).max() <= 1e-9 * np.abs(p).max()


def test_more_neighbours_than_a_record_names():
    """Vertex 0 in a hinge with every three of the others, in each place in turn, and in a triangle with the last two:
    its block against the oracle's. Both sum 700,000 terms of random sign in FP64 in different orders, which leaves
    1e-16 * sqrt(700,000) = 1e-13 of the sum of their sizes; the 21 highest neighbours, those that no place names,
    are in seven hinges and the triangle and carry 1e-5 of it."""
    n = PLACES + 20 + (PLACES + 20 + 2) % 3  # others in threes
    assert (n - 1) % 3 == 0 and n - 1 > PLACES
    rng = np.random.default_rng(9)
    others = np.arange(1, n, dtype=np.uint32).reshape(-1, 3)
    others[-1] = others[-1][::-1]
    H = len(others)
    hinges = np.zeros((H, 4), np.uint32)
    for slot in range(4):
        rows = np.arange(H) % 4 == slot
        hinges[np.ix_(rows, [c for c in range(4) if c != slot])] = others[rows]
    uv = rng.uniform(-1.0, 1.0, (n, 2))
    uv[0], uv[n - 2], uv[n - 1] = (0.0, 0.0), (0.01, 0.0), (0.0, 0.01)
    tri = np.array([[0, n - 2, n - 1]], np.uint32)
    inv_dm, area = scenes.inverse_rest(uv, tri.astype(np.int64))
    mesh = scenes.Mesh(
        uv=uv, triangles=tri, inv_dm=inv_dm, area=area, triangle_material=np.zeros(1, np.uint32), hinges=hinges,
        hinge_weight=np.ones(H), hinge_across=np.tile([1.0, 0.0], (H, 1)), hinge_material=np.zeros(H, np.uint32),
        materials=[scenes.Material()], rest_area=np.ones(n), masses=np.full(n, 1e-3), pinned=np.zeros(n, np.uint8),
        pin_positions=np.zeros((n, 3)))
    x = np.stack([uv[:, 0], rng.uniform(0.5, 1.5, n), uv[:, 1]], axis=1)
    x[0], x[n - 2], x[n - 1] = (0.0, 0.0, 0.0), (0.011, 0.001, 0.0), (0.0, 0.0, 0.009)
    sc = scenes.Scene("hub", mesh, None, x, np.zeros_like(x), scenes.StepSettings(dt=1 / 60, radius=0.001, stiffness=1e4), 1)
    st = sc.settings.to_c()
    eg, gg, hg = VbdSolver(sc).local_blocks(x, 0.002, st)
    eo, go, ho = oracle.Solver(sc, threads=8).local_blocks(x, 0.002, st)
    assert abs(eg[0] - eo[0]) <= 1e-10 * eo[0]
    assert np.all(np.abs(gg[0] - go[0]) <= 1e-8 * np.abs(go[0]).max())
    assert np.all(np.abs(hg[0] - ho[0]) <= 1e-8 * np.abs(ho[0]).max())
    assert np.all(np.abs(eg[1:] - eo[1:]) <= 1e-9 * np.abs(eo[1:]).max())
