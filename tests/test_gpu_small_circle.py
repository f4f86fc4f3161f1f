"""A circle smaller than the exit rule's shift (and 5e-4, the least distance
from its centre that the rule knows): paths go on near the centre, where the
normal and with it the shift shrink, and stop elsewhere.  FP64 paths follow
the oracle's, with lane groups and without, for a subdomain and a domain."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SEED = 20251203


@pytest.mark.parametrize("problem,cv", [(0, 0), (0, 1), (2, 0), (2, 1), (3, 0)])
@pytest.mark.parametrize("r", [1.0e-3, 1.2e-3, 4e-4])
def test_small_circle_matches_oracle(gpu, orc, fk, problem, cv, r):
    h, n, x, y = 1e-6, 3000, 0.4, 0.45  # a step of 1e-3, a shift of 8e-4 or a little less
    disk = problem == fk.DISK
    dom, prob = ((r, x, y), (0.5, 0.5, 0.5, 0)) if disk else ((0, 0, 1, 1), (0, 0, 0, 0))
    b = gpu.register_bvp(problem, cv=cv, dom=dom, prob=prob)
    kw = {} if disk else dict(sub_shape=[1], sub_params=np.array([[r, x, y, 0.0]]))
    gpu.set_stream(81)
    st = gpu.solve_points(b, np.array([[x, y]]), n, h, fk.FP64, **kw)
    ob = orc.bvp(problem, cv=cv, dom=dom, dom_shape=fk.CIRCLE if disk else fk.RECT, prob=prob)
    o = orc.Session(orc.RNG_PHILOX, seed=SEED, stream=81).point_solve(ob, x, y, n, h, item=0,
                                                                    sub=None if disk else orc.shape(1, (r, x, y, 0.0)))
    for k in orc.STAT_NAMES:
        assert np.isclose(st[k][0], o[k], rtol=1e-9, atol=1e-12), (k, st[k][0], o[k])
    if r < 5e-4:
        assert st["mean_steps"][0] == 1
    else:
        assert 1.01 < st["mean_steps"][0] < 1.5


@pytest.mark.parametrize("problem", [0, 2])
def test_small_circle_beside_the_domain(gpu, orc, fk, problem):
    """The centre lies within the shift of a side of the domain: the nearer of the
    two boundaries decides alone."""
    h, n, x, y, r = 1e-6, 3000, 9e-4, 0.45, 1.2e-3
    b = gpu.register_bvp(problem)
    gpu.set_stream(82)
    st = gpu.solve_points(b, np.array([[x, y]]), n, h, fk.FP64, sub_shape=[1], sub_params=np.array([[r, x, y, 0.0]]))
    o = orc.Session(orc.RNG_PHILOX, seed=SEED, stream=82).point_solve(orc.bvp(problem), x, y, n, h, item=0,
                                                                    sub=orc.shape(1, (r, x, y, 0.0)))
    for k in orc.STAT_NAMES:
        assert np.isclose(st[k][0], o[k], rtol=1e-9, atol=1e-12), (k, st[k][0], o[k])
    assert 1.01 < st["mean_steps"][0] < 1.5 and 0 < st["n_domain_exits"][0] < n
