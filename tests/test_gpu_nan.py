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


@pytest.mark.parametrize("n", [1, 200, 5000])
def test_a_sum_that_overflows_is_infinite(fk, n):
    """A start point so far below the square that the source is 1e301 per step:
    the mean is finite, the mean square overflows and says so."""
    r = _solve(fk, fk.FRANKE, (0, 0, 1, 1), [[0.5, -780.0], [0.5, 0.5]], 1e-3, n, 100000)
    assert np.isfinite(r["phi"][0]) and abs(r["phi"][0]) > 1e290
    assert np.isposinf(r["phiphi"][0]) and np.isfinite(r["phiphi"][1])


def test_nan_disk_leaves_the_others_of_its_batch(gpu, fk):
    """A disk with a NaN grid angle, before and between sound ones of several
    angles: each of these gets the rows that it gets alone.  (Franke: the
    operators hold no NaN.)"""
    b = gpu.register_bvp(fk.FRANKE)
    disks = []
    for i, t0 in enumerate([NAN, 0.3, 0.1, NAN, 0.2, 0.1, 0.3, 0.2]):
        th = 2 * np.pi * np.arange(16) / 16
        c = np.array([0.4 + 0.02 * i, 0.5])
        disks.append(dict(cx=c[0], cy=c[1], radius=0.1, theta0=t0, n_circle=16, n_radial=11, periph_theta=th,
                          inner_xy=np.stack([c[0] + 0.05 * np.cos([0.2, 1.3]), c[1] + 0.05 * np.sin([0.2, 1.3])], 1)))
    for d, (G, B) in zip(disks, gpu.solve_disks_ps(b, disks)):
        if not np.isnan(d["theta0"]):
            (g, v), = gpu.solve_disks_ps(b, [d])
            assert np.isfinite(g).all() and np.array_equal(G, g) and np.array_equal(B, v)


def test_nan_disk_operators_leave_the_others_of_their_batch(gpu, fk):
    """A disk whose mode matrices hold NaN (varying c at a NaN centre): its
    elimination stays in its rows, the other disks get theirs."""
    b = gpu.register_bvp(fk.ANISO)
    disks = []
    for i, cx in enumerate([0.4, NAN, 0.5, NAN]):
        th = 0.1 + 2 * np.pi * np.arange(16) / 16
        c = np.array([cx, 0.5])
        disks.append(dict(cx=c[0], cy=c[1], radius=0.1, theta0=0.1, n_circle=16, n_radial=11, periph_theta=th,
                          inner_xy=np.stack([c[0] + 0.05 * np.cos([0.2, 1.3]), c[1] + 0.05 * np.sin([0.2, 1.3])], 1)))
    for d, (G, B) in zip(disks, gpu.solve_disks_ps(b, disks)):
        if not np.isnan(d["cx"]):
            (g, v), = gpu.solve_disks_ps(b, [d])
            assert np.isfinite(g).all() and np.array_equal(G, g) and np.array_equal(B, v)
