"""FP64 stepping's fixed-point functions and lean exit test at the edges of
their ranges, against the oracle on the same stream (the same paths: rtol
1e-9, as in test_gpu_parity)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SEED = 20251203

# the fixed-point range is [-3/8, 11/8) in each coordinate: domains inside it, across its edges and far outside
CASES = {
    "across_edges": (0, 0, (-1, -1, 2, 2), [(-0.375, 0.5), (1.375, 1.374), (0.4, -0.38), (1.9, 1.9)], None, 2e-3),
    "across_edges_aniso_cv": (2, 1, (-1, -1, 2, 2), [(-0.3749, 0.2), (1.36, -0.37), (0.5, 1.4)], None, 2e-3),
    "far_outside": (0, 1, (5, 5, 6, 6), [(5.4, 5.5)], None, 1e-3),
    "far_outside_aniso": (2, 0, (-4, 2, -3, 3), [(-3.4, 2.5)], None, 1e-3),
    "start_outside_domain": (0, 0, (0, 0, 1, 1), [(1.2, 0.5), (-0.1, -0.1)], None, 1e-3),
    "large_step": (2, 0, (0, 0, 1, 1), [(0.5, 0.5), (0.01, 0.99)], None, 0.05),
    "small_step": (0, 0, (0, 0, 0.02, 0.02), [(0.01, 0.011)], None, 1e-7),
    "rect_inside_domain": (2, 1, (0, 0, 1, 1), [(0.3, 0.3)], (0, (0.2, 0.25, 0.45, 0.4)), 5e-4),
    "rect_sharing_sides": (2, 0, (0, 0, 1, 1), [(0.05, 0.06)], (0, (0.0, 0.0, 0.15, 0.2)), 5e-4),
    "rect_over_domain": (0, 0, (0, 0, 1, 1), [(0.95, 0.9)], (0, (0.8, 0.7, 1.3, 1.2)), 5e-4),
    "circle_over_domain": (0, 1, (0, 0, 1, 1), [(0.1, 0.1), (0.02, 0.3)], (1, (0.25, 0.1, 0.15, 0.0)), 5e-4),
    "circle_below_threshold": (0, 0, (0, 0, 1, 1), [(0.5, 0.5)], (1, (0.01, 0.5, 0.5, 0.0)), 1e-3),
    "disk": (3, 1, (0.7, 1.5, -2.0), [(1.4, -1.9), (1.5, -2.0), (2.1, -2.2)], None, 1e-3),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_point_solves_match_oracle(gpu, orc, fk, name):
    problem, cv, dom, pts, sub, h = CASES[name]
    prob = (dom[1], dom[2], dom[0], 0) if problem == fk.DISK else (0, 0, 0, 0)
    b = gpu.register_bvp(problem, cv=cv, dom=dom, prob=prob)
    N = 700
    gpu.set_stream(900)
    kw = {}
    if sub is not None:
        kw = dict(sub_shape=[sub[0]] * len(pts), sub_params=np.tile(sub[1], (len(pts), 1)))
    st = gpu.solve_points(b, np.array(pts), N, h, fk.FP64, **kw)
    s = orc.Session(orc.RNG_PHILOX, seed=SEED)
    s.set_stream(900)
    ob = orc.bvp(problem, cv=cv, dom=dom, dom_shape=fk.CIRCLE if problem == fk.DISK else fk.RECT, prob=prob)
    for i, (x, y) in enumerate(pts):
        o = s.point_solve(ob, x, y, N, h, item=i, sub=orc.shape(sub[0], sub[1]) if sub is not None else None)
        for k in orc.STAT_NAMES:
            assert np.isclose(st[k][i], o[k], rtol=1e-9, atol=1e-12), (k, i, st[k][i], o[k])
