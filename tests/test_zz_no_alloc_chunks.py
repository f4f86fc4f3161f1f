"""fk_solve_points_noalloc spreads its paths over the warps of the grid: about
the path kernel's time of the allocating call, for few paths and many, one
point and many.  (Anisotropic problem: no lane groups on either side.)"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SEED = 20251203


@pytest.mark.parametrize("precision,n,paths", [("FP32", 1, 4_000_000), ("FP32", 1024, 10_000), ("FP32", 37, 1501), ("FP64", 1, 20_000),
                                               ("FP64", 1, 1000), ("FP32", 3, 300_001)])
def test_noalloc_time_and_results(fk, precision, n, paths):
    """Bound: a quarter more (its grid does not follow the number of paths, which
    the host does not know), and 0.15 ms for the prepare and finalize launches
    and the memsets, which the allocating call's kernel time leaves out."""
    import torch
    L, prec, h, sid = fk.load(), getattr(fk, precision), 1e-3, 31
    pts = np.random.default_rng(6).uniform(0.2, 0.8, (n, 2))
    ctx = fk.Context(device=0, seed=SEED)
    try:
        b = ctx.register_bvp(fk.ANISO)
        t_ref = 1e30
        for _ in range(5):
            ctx.set_stream(sid)
            ref = ctx.solve_points(b, pts, paths, h, prec)
            t_ref = min(t_ref, ctx.last_timing()[0])
    finally:
        ctx.close()
    d = fk.BvpDesc()
    d.problem, d.cv, d.dom_shape, d.mlp_id = fk.ANISO, fk.CV_NONE, fk.RECT, -1
    d.dom[2] = d.dom[3] = 1.0
    xy = torch.tensor(pts, dtype=torch.float64, device="cuda")
    p = torch.full((n,), paths, dtype=torch.int32, device="cuda")
    hh = torch.full((n,), h, dtype=torch.float64, device="cuda")
    out = torch.zeros((n, len(fk.STAT_FIELDS)), dtype=torch.float64, device="cuda")
    ptr = [C.c_void_p(v.data_ptr()) for v in (xy, p, hh, out)]
    s = torch.cuda.current_stream()
    best = 1e30
    for _ in range(7):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(s)
        rc = L.fk_solve_points_noalloc(C.byref(d), SEED, sid, n, ptr[0], ptr[1], ptr[2], prec, 1 << 24, C.c_void_p(s.cuda_stream), ptr[3])
        e1.record(s)
        assert rc == fk.FK_OK
        e1.synchronize()
        best = min(best, e0.elapsed_time(e1))
    got = out.cpu().numpy()
    for j, name in enumerate(fk.STAT_FIELDS):
        assert np.allclose(got[:, j], ref[name], rtol=1e-6, atol=1e-12), name
    assert best <= 1.25 * t_ref + 0.15, (best, t_ref)


def test_noalloc_sums_keep_their_roundings(fk):
    """FP64 sums' roundings lie in the output records until the end of the call,
    whatever was there before: sums of squares as from fk_solve_points (the two
    calls' parts differ, their roundings average out, the total's and the mean's
    are 2^-53 / sqrt 3 each on either side: 1.2 times 2^-53 between the calls)."""
    import torch
    L, n, paths, h, sid = fk.load(), 1000, 2000, 1e-3, 32
    pts = np.random.default_rng(7).uniform(0.1, 0.9, (n, 2))
    ctx = fk.Context(device=0, seed=SEED)
    try:
        ctx.set_stream(sid)
        ref = ctx.solve_points(ctx.register_bvp(fk.ANISO), pts, paths, h, fk.FP64)
    finally:
        ctx.close()
    d = fk.BvpDesc()
    d.problem, d.cv, d.dom_shape, d.mlp_id = fk.ANISO, fk.CV_NONE, fk.RECT, -1
    d.dom[2] = d.dom[3] = 1.0
    xy = torch.tensor(pts, dtype=torch.float64, device="cuda")
    p = torch.full((n,), paths, dtype=torch.int32, device="cuda")
    hh = torch.full((n,), h, dtype=torch.float64, device="cuda")
    out = torch.full((n, len(fk.STAT_FIELDS)), float("nan"), dtype=torch.float64, device="cuda")
    s = torch.cuda.current_stream()
    ptr = [C.c_void_p(v.data_ptr()) for v in (xy, p, hh, out)]
    assert L.fk_solve_points_noalloc(C.byref(d), SEED, sid, n, ptr[0], ptr[1], ptr[2], fk.FP64, 1 << 24, C.c_void_p(s.cuda_stream),
                                     ptr[3]) == fk.FK_OK
    torch.cuda.synchronize()
    got = dict(zip(fk.STAT_FIELDS, out.cpu().numpy().T))
    e = (got["phiphi"] - ref["phiphi"]) / ref["phiphi"]
    assert np.sqrt(np.mean(e * e)) <= 2.0 ** -52, np.sqrt(np.mean(e * e))
    assert np.array_equal(got["n_paths"], ref["n_paths"]) and np.array_equal(got["mean_steps"], ref["mean_steps"])
