"""Schedules of the path kernel that a call's size picks: a group of 8 or 32
lanes per path (FP64, constant coefficients), streaming of chunks of one class
and of several (point solves), fewer warps for few paths.  FP64 results equal
the oracle's per item (the same paths: rtol 1e-9) and those of a caller-set
launch shape, which takes a lane per path."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SEED = 20251203
FAR = (-200, -200, 200, 200)


def _against_oracle(orc, st, i, ob, x, y, n, h, stream, sub=None):
    s = orc.Session(orc.RNG_PHILOX, seed=SEED, stream=stream)
    o = s.point_solve(ob, x, y, int(n), h, item=i, sub=sub)
    for k in orc.STAT_NAMES:
        assert np.isclose(st[k][i], o[k], rtol=1e-9, atol=1e-12), (k, i, st[k][i], o[k])
    assert st["n_paths"][i] == n


# n paths: less than a group's, ragged over 8 and 32 lanes, several chunks; the
# last two have the size and step at which 8 lanes per path are picked
@pytest.mark.parametrize("n,h", [(1, 1e-3), (3, 1e-3), (33, 1e-3), (1001, 1e-3), (100003, 4e-3), (60001, 3e-3)])
@pytest.mark.parametrize("problem,cv,dom,sub", [
    (0, 0, (0, 0, 1, 1), None), (0, 1, (0, 0, 1, 1), (1, (0.3, 0.5, 0.5, 0))), (1, 1, FAR, (0, (-72.3, -38.2, -71.75, -37.7))),
    (3, 0, (0.6, -71.9, -38.1), None), (5, 0, FAR, (1, (0.5, -72.0, -38.0, 0)))])
def test_lane_groups_match_oracle(gpu, orc, fk, problem, cv, dom, sub, n, h):
    prob = (dom[1], dom[2], dom[0], 0) if problem == fk.DISK else (0, 0, 0, 0)
    xy = np.array([[0.45, 0.55]]) if problem == 0 else np.array([[-72.0, -38.0]])
    b = gpu.register_bvp(problem, cv=cv, dom=dom, prob=prob)
    kw = {} if sub is None else dict(sub_shape=[sub[0]], sub_params=np.array([sub[1]], dtype=float))
    gpu.set_stream(71)
    st = gpu.solve_points(b, xy, n, h, fk.FP64, **kw)
    ob = orc.bvp(problem, cv=cv, dom=dom, dom_shape=fk.CIRCLE if problem == fk.DISK else fk.RECT, prob=prob)
    _against_oracle(orc, st, 0, ob, *xy[0], n, h, 71, orc.shape(sub[0], sub[1]) if sub else None)


@pytest.mark.parametrize("problem", [0, 1])
def test_lane_groups_step_cap(gpu, fk, problem):
    """Paths cut at max_steps, inside a round of a group and at its end."""
    dom = (0, 0, 1, 1) if problem == 0 else FAR
    xy = np.array([[0.5, 0.5], [0.1, 0.2]]) if problem == 0 else np.array([[0.0, 0.0], [10.0, -3.0]])
    b = gpu.register_bvp(problem, dom=dom)
    for cap in (1, 5, 32, 33, 64):
        out = []
        for shape in (0, 128):
            gpu.set_launch(256 if shape else 0, shape)
            gpu.set_max_steps(cap)
            gpu.set_stream(72)
            out.append(gpu.solve_points(b, xy, 500, 1e-4, fk.FP64, allow=(fk.FK_ERR_STEP_CAP,)))
        gpu.set_launch(0, 0)
        gpu.set_max_steps(1 << 24)
        assert out[0]["n_capped"].sum() > 0
        for k in out[0]:
            assert np.allclose(out[0][k], out[1][k], rtol=1e-11, atol=1e-13), (cap, k)


@pytest.mark.parametrize("classes", [1, 2, 7, 300])
@pytest.mark.parametrize("problem", [0, 2])
def test_streaming_matches_oracle(gpu, orc, fk, problem, classes):
    """Items of 0 to a few hundred paths whose step sizes fall into one class,
    several, and more than are told apart; a caller-set launch shape keeps a
    lane per path."""
    rng = np.random.default_rng(classes)
    n = 311
    xy = rng.uniform(0.05, 0.95, (n, 2))
    paths = np.where(rng.random(n) < 0.1, 0, rng.integers(1, 260, n)).astype(np.uint32)
    h = (1e-3 * (1 + 0.01 * np.arange(classes)))[rng.integers(0, classes, n)]
    b = gpu.register_bvp(problem)
    ob = orc.bvp(problem)
    for shape in ((0, 0), (64, 40)):
        gpu.set_launch(*shape)
        gpu.set_stream(73)
        st = gpu.solve_points(b, xy, paths, h, fk.FP64)
        gpu.set_launch(0, 0)
        assert np.array_equal(st["n_paths"], paths)
        for i in list(range(0, n, 29)):
            if paths[i]:
                _against_oracle(orc, st, i, ob, *xy[i], paths[i], h[i], 73)


@pytest.mark.parametrize("classes", [1, 5])
def test_streaming_fp32_pairs_with_fp64(gpu, fk, classes):
    rng = np.random.default_rng(5)
    n = 400
    xy = rng.uniform(0.05, 0.95, (n, 2))
    paths = rng.integers(1, 900, n).astype(np.uint32)
    h = (1e-3 * (1 + 0.1 * np.arange(classes)))[rng.integers(0, classes, n)]
    b = gpu.register_bvp(fk.ANISO, cv=fk.CV_EXACT)
    st = []
    for prec in (fk.FP64, fk.FP32):
        gpu.set_stream(74)
        st.append(gpu.solve_points(b, xy, paths, h, prec))
    assert np.array_equal(st[1]["n_paths"], paths)
    # a path whose last FP32 position rounds across the threshold stops a step apart: about 1e-6 of the paths
    same = st[0]["RNGC"] == st[1]["RNGC"]
    assert same.mean() > 0.99
    for k in ("phi", "phiphi", "phi_VR", "phiphi_VR", "xiphi", "xi_sq_mean"):
        assert np.allclose(st[0][k][same], st[1][k][same], rtol=2e-4, atol=2e-4), k


@pytest.mark.parametrize("precision", ["FP64", "FP32"])
def test_patch_stencil_streaming_rows(gpu, fk, precision):
    """Few paths per item on a patch mesh (FP64 streams through the items of a
    patch; FP32 forms its rows per item): the same G and B as in slot mode."""
    mesh = gpu.mesh_square_patches((0, 0, 1, 1), 3, 15, 0.25, 1.0, 20)
    b = gpu.register_bvp(fk.ANISO)
    prec = getattr(fk, precision)
    out = []
    for shape in ((0, 0), (256, 512)):
        gpu.set_launch(*shape)
        gpu.set_stream(75)
        out.append(gpu.assemble(mesh, b, 333, 5e-4, prec))
    gpu.set_launch(0, 0)
    tol = 1e-11 if precision == "FP64" else 2e-6
    for k in ("val", "B", "item_G", "item_B"):
        assert np.allclose(out[0][k], out[1][k], rtol=tol, atol=tol), k


@pytest.mark.parametrize("problem", [0, 2])
def test_disk_rows_shared_operators(gpu, fk, problem):
    """A batch whose disks share radii, grids and periphery angles in part gives
    each disk the rows that it gets alone, bit for bit."""
    rng = np.random.default_rng(3)
    disks = []
    for i in range(12):
        nc, r, t0 = (16, 20)[i % 3 == 2], (0.1, 0.17)[i % 2], (0.1, 0.3)[i % 4 == 3]
        c = rng.uniform(0.3, 0.7, 2)
        th = t0 + 2 * np.pi * np.arange(nc) / nc
        if i == 7:
            th = th + 1e-3
        rr, aa = 0.9 * r * np.sqrt(rng.random(5)), 2 * np.pi * rng.random(5)
        disks.append(dict(cx=c[0], cy=c[1], radius=r, theta0=t0, n_circle=nc, n_radial=(11, 13)[i % 5 == 4], periph_theta=th,
                          inner_xy=np.stack([c[0] + rr * np.cos(aa), c[1] + rr * np.sin(aa)], 1)))
    b = gpu.register_bvp(problem)
    batch = gpu.solve_disks_ps(b, disks)
    for d, (G, B) in zip(disks, batch):
        (g, v), = gpu.solve_disks_ps(b, [d])
        assert np.array_equal(G, g) and np.array_equal(B, v)
