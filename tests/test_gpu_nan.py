"""Non-finite input where an entry point takes it: a call ends as the exit rule
says, and what is not NaN itself stays as it is."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solve(fk, problem, dom, xy, h, n, cap, cv=0, prob=(0, 0, 0, 0)):
    """fk_solve_points_noalloc (whose coordinates lie on the device and are not checked), FP64."""
    import torch
    L = fk.load()
    d = fk.BvpDesc()
    d.problem, d.cv, d.mlp_id = problem, cv, -1
    d.dom_shape = fk.CIRCLE if problem == fk.DISK else fk.RECT
    for i, v in enumerate(dom):
        d.dom[i] = v
    for i, v in enumerate(prob):
        d.prob[i] = v
    t = torch.tensor(xy, dtype=torch.float64, device="cuda")
    p = torch.full((len(xy),), n, dtype=torch.int32, device="cuda")
    hh = torch.full((len(xy),), h, dtype=torch.float64, device="cuda")
    out = torch.zeros((len(xy), len(fk.STAT_FIELDS)), dtype=torch.float64, device="cuda")
    s = torch.cuda.current_stream()
    ptr = [C.c_void_p(v.data_ptr()) for v in (t, p, hh, out)]
    rc = L.fk_solve_points_noalloc(C.byref(d), 77, 5, len(xy), ptr[0], ptr[1], ptr[2], fk.FP64, cap, C.c_void_p(s.cuda_stream),
                                   ptr[3])
    assert rc == fk.FK_OK
    torch.cuda.synchronize()
    return dict(zip(fk.STAT_FIELDS, out.cpu().numpy().T))


NAN = float("nan")


def test_nan_abscissa_in_a_rectangle_leaves_the_ordinate(fk):
    """rect_dist of a NaN abscissa is the other offset: the path stops where its
    ordinate does, as in a domain whose other sides are far away."""
    r = _solve(fk, fk.FRANKE, (0, 0, 1, 1), [[NAN, 0.5], [0.4, 0.3]], 1e-3, 200, 100000)
    w = _solve(fk, fk.FRANKE, (-1e6, 0, 1e6, 1), [[0.5, 0.5], [0.4, 0.3]], 1e-3, 200, 100000)
    assert r["mean_steps"][0] == w["mean_steps"][0] > 10 and r["n_capped"][0] == 0 and r["n_paths"][0] == 200
    assert np.isnan(r["phi"][0]) and np.isfinite(r["phi"][1])


def test_nan_ordinate_stops_at_once(fk):
    r = _solve(fk, fk.FRANKE, (0, 0, 1, 1), [[0.5, NAN]], 1e-3, 200, 1000)
    assert r["mean_steps"][0] == 1 and np.isnan(r["phi"][0])


@pytest.mark.parametrize("xy", [(NAN, 0.5), (0.5, NAN), (float("inf"), 0.5)])
def test_nan_sigma_stops_at_once(fk, xy):
    """sigma at a non-finite point is NaN, and so is the threshold."""
    r = _solve(fk, fk.ANISO, (0, 0, 1, 1), [list(xy)], 1e-3, 200, 1000)
    assert r["mean_steps"][0] == 1 and np.isnan(r["phi"][0]) and r["n_paths"][0] == 200


def test_nan_in_a_circle_stops_at_once(fk):
    """The normal of a NaN position is NaN, and with it the threshold."""
    r = _solve(fk, fk.DISK, (0.6, 0.0, 0.0), [[NAN, 0.1], [0.1, 0.1]], 1e-3, 100, 50, prob=(0.0, 0.0, 0.6, 0))
    assert r["n_capped"][0] == 0 and r["mean_steps"][0] == 1 and np.isnan(r["phi"][0])
    assert np.isfinite(r["phi"][1])
