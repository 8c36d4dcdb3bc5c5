"""The scenes of the closed-form comparison (test_gpu_terms.py) reach every kind
of contact within its radius, mollified edge pairs and the logarithmic part of the
activation. On the CPU, from the oracle's contacts."""
import numpy as np

import oracle
import test_gpu_terms


def distance(kind, p):
    if kind == 0:
        return np.linalg.norm(p[0] - p[1])
    if kind == 1:
        u, w = p[2] - p[1], p[0] - p[1]
        return np.linalg.norm(w - u * (w @ u) / (u @ u))
    n = np.cross(p[2] - p[1], p[3] - p[1]) if kind == 2 else np.cross(p[1] - p[0], p[3] - p[2])
    return abs((p[0] - p[1 if kind == 2 else 2]) @ n) / np.linalg.norm(n)


def test_every_kind_is_active_somewhere():
    marks = [m for m in test_gpu_terms.test_blocks_match_forward_differentiation.pytestmark if m.name == "parametrize"]
    kinds, mollified, logarithmic = set(), 0, 0
    for shift, turn, gap, jitter, material in marks[0].args[1]:
        for seed in range(3):
            sc = test_gpu_terms.two_layers(shift, turn, gap, jitter, material, seed)
            r = sc.settings.radius
            c = oracle.World(sc.x0, sc.mesh.triangles, sc.n).detect(sc.x0, 0.004, sc.settings.ogc_c())
            for kind, v, eps in zip(c["kinds"], c["vertices"], c["epsilon"]):
                p = sc.x0[v]
                d = distance(kind, p)
                if d >= r:
                    continue
                kinds.add(int(kind))
                logarithmic += d < 0.5 * r
                if kind == 3:
                    n = np.cross(p[1] - p[0], p[3] - p[2])
                    mollified += n @ n < eps
    assert kinds == {0, 1, 2, 3} and mollified > 0 and logarithmic > 0, (kinds, mollified, logarithmic)
