"""Which schedule a call gets (fk_last_schedule): lanes per path and streaming
by the call's size, and the launch shape that its caller set."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SEED = 20251203


# FP64, Franke on the unit square from (0.45, 0.55): paths, step, lanes per path
@pytest.mark.parametrize("n,h,lanes", [(1, 1e-3, 32), (1001, 1e-3, 32), (60001, 3e-3, 32), (100003, 4e-3, 8), (300000, 1e-2, 8),
                                       (1000000, 1e-2, 1)])
def test_lanes_per_path(gpu, orc, fk, n, h, lanes):
    b = gpu.register_bvp(fk.FRANKE)
    gpu.set_stream(171)
    st = gpu.solve_points(b, np.array([[0.45, 0.55]]), n, h, fk.FP64)
    s = gpu.last_schedule()
    assert s["lanes"] == lanes and s["streaming"] == (1 if lanes == 1 else 0)
    if n <= 100003:
        o = orc.Session(orc.RNG_PHILOX, seed=SEED, stream=171).point_solve(orc.bvp(fk.FRANKE), 0.45, 0.55, n, h, item=0)
        for k in orc.STAT_NAMES:
            assert np.isclose(st[k][0], o[k], rtol=1e-9, atol=1e-12), k


@pytest.mark.parametrize("problem,precision,paths,streaming", [(2, "FP64", 1000, 1), (2, "FP64", 5000, 1), (2, "FP32", 1000, 0),
                                                               (2, "FP32", 5000, 1), (0, "FP32", 1000, 0)])
def test_streaming_by_paths_per_item(gpu, fk, problem, precision, paths, streaming):
    """FP64 points whose coefficients vary stream, FP32 points from 3,072 paths an item on."""
    b = gpu.register_bvp(problem)
    xy = np.random.default_rng(1).uniform(0.1, 0.9, (40, 2))
    gpu.solve_points(b, xy, paths, 1e-3, getattr(fk, precision))
    s = gpu.last_schedule()
    assert s["lanes"] == 1 and s["streaming"] == streaming and s["classes"] == 1
    gpu.solve_points(b, xy, paths, np.where(np.arange(40) % 4 == 0, 1e-3, 2e-3), getattr(fk, precision))
    assert gpu.last_schedule()["classes"] == (2 if streaming else 1)


@pytest.mark.parametrize("block", [32, 64, 128, 256])
@pytest.mark.parametrize("n,h,lanes", [(1001, 1e-3, 32), (100003, 4e-3, 8), (1000000, 1e-2, 1)])
def test_callers_block_is_kept(gpu, fk, block, n, h, lanes):
    """Whichever kernel runs, and with the default's results."""
    b = gpu.register_bvp(fk.FRANKE)
    out = []
    for shape in (0, block):
        gpu.set_launch(shape, 0)
        gpu.set_stream(172)
        out.append(gpu.solve_points(b, np.array([[0.45, 0.55]]), n, h, fk.FP64))
        s = gpu.last_schedule()
        gpu.set_launch(0, 0)
        assert s["lanes"] == lanes
    assert s["block"] == block and s["grid"] > 0
    assert out[1]["n_paths"][0] == n
    for k in out[0]:
        assert np.allclose(out[0][k], out[1][k], rtol=1e-11, atol=1e-13), k


# the last: FP32, more paths than the machine has lanes for
@pytest.mark.parametrize("problem,precision,n,paths,h", [(0, "FP64", 1, 1000, 1e-3), (0, "FP64", 64, 4000, 1e-3), (2, "FP64", 37, 1501, 1e-3),
                                                         (3, "FP64", 5, 20000, 1e-3), (2, "FP32", 256, 10000, 1e-3)])
def test_tuned_shape_keeps_the_lanes_of_the_size(gpu, fk, problem, precision, n, paths, h):
    """The autotuner times shapes of the schedule that the tuned call runs: its
    lanes per path are the untuned call's, and so are its results."""
    dom, prob = ((0.5, 0.5, 0.5), (0.5, 0.5, 0.5, 0)) if problem == fk.DISK else ((0, 0, 1, 1), (0, 0, 0, 0))
    b = gpu.register_bvp(problem, dom=dom, prob=prob)
    xy = np.random.default_rng(2).uniform(0.3, 0.7, (n, 2))
    ids, p, hh = np.full(n, b, dtype=np.int32), np.full(n, paths, dtype=np.uint32), np.full(n, h)
    prec = getattr(fk, precision)
    out = []
    for tune in (False, True):
        gpu.set_launch(0, 0)
        if tune:
            block, chunk, _ = gpu.autotune_points(ids, xy, p, hh, prec, sample_fraction=0.25)
        gpu.set_stream(173)
        out.append((gpu.solve_points_multi(ids, xy, p, hh, prec), gpu.last_schedule()))
    gpu.set_launch(0, 0)
    s = out[1][1]
    assert s["lanes"] == out[0][1]["lanes"] and s["block"] == block
    assert s["chunk"] == max(32, chunk // (block // 32)) // s["lanes"]  # the warps of a block share a chunk, a path counts as its lanes
    tol = 1e-11 if precision == "FP64" else 1e-6
    for k in out[0][0]:
        assert np.allclose(out[0][0][k], out[1][0][k], rtol=tol, atol=tol), k


@pytest.mark.parametrize("shape", [(256, 8192), (64, 8192), (256, 40), (32, 7)])
def test_callers_chunk_is_the_blocks(gpu, fk, shape):
    """A point solve's warps take the caller's chunk in parts, a lane per path."""
    b = gpu.register_bvp(fk.FRANKE)
    gpu.set_launch(*shape)
    st = gpu.solve_points(b, np.array([[0.4, 0.5], [0.6, 0.6]]), 5000, 1e-3, fk.FP64)
    s = gpu.last_schedule()
    gpu.set_launch(0, 0)
    assert s["lanes"] == 1 and s["chunk"] == max(min(shape[1], 32), shape[1] // (shape[0] // 32))
    assert (st["n_paths"] == 5000).all()


@pytest.mark.parametrize("precision", ["FP64", "FP32"])
@pytest.mark.parametrize("problem", [0, 2])
@pytest.mark.parametrize("paths", [20, 33, 64])
def test_arc_rows_of_few_paths_repeat(gpu, fk, problem, precision, paths):
    """The rows of items of up to 64 paths are the same in every run, though the
    inverse of a 44-node arc turns a rounding of a moment into 1e-7 of a row."""
    mesh = gpu.mesh_circles((0, 0, 1, 1), 4, 1.2, 0.121, 44)
    b = gpu.register_bvp(problem)
    out = []
    for _ in range(3):
        gpu.set_stream(174)
        out.append(gpu.assemble(mesh, b, paths, 1e-4, getattr(fk, precision)))
    for r in out[1:]:
        assert np.array_equal(r["item_G"], out[0]["item_G"])


def test_fp64_sums_do_not_depend_on_their_parts(gpu, fk):
    """1,000 points of 2,000 paths in chunks of 64 and of 32 paths, which reach an
    item's sums in a few hundred parts (chunks, and paths that outlive them).  The
    sums of squares of the two runs hold the same terms; the roundings of the parts
    average out, the total's and the mean's do not: on either side 2^-53 / sqrt 3
    each, sqrt(4 / 3) = 1.2 times 2^-53 between the runs.  (Parts rounded to the
    whole one after the other: about 4 times 2^-53.)"""
    b = gpu.register_bvp(fk.ANISO)
    xy = np.random.default_rng(7).uniform(0.1, 0.9, (1000, 2))
    out = []
    for shape in ((0, 0), (32, 32)):
        gpu.set_launch(*shape)
        gpu.set_stream(175)
        out.append(gpu.solve_points(b, xy, 2000, 1e-3, fk.FP64)["phiphi"])
    gpu.set_launch(0, 0)
    d = (out[0] - out[1]) / out[0]
    assert np.sqrt(np.mean(d * d)) <= 2.0 ** -52, np.sqrt(np.mean(d * d)) * 2.0 ** 53


@pytest.mark.parametrize("paths,block,chunk,part", [(1 << 20, 256, 8192, 1024), (1 << 20, 256, 512, 64), (1 << 20, 32, 16, 16),
                                                    (100_000_000, 256, 512, 95), (100_000_000, 256, 8192, 1024)])
def test_parts_of_a_callers_chunk(gpu, fk, paths, block, chunk, part):
    """A warp takes its part of the caller's chunk, but the host lists no more than
    2^20 parts for it (100 M paths >> 20 = 95)."""
    b = gpu.register_bvp(fk.FRANKE)
    gpu.set_launch(block, chunk)
    st = gpu.solve_points(b, np.array([[0.05, 0.05]]), paths, 1e-2, fk.FP32)
    s = gpu.last_schedule()
    gpu.set_launch(0, 0)
    assert s["chunk"] == part and s["block"] == block and st["n_paths"][0] == paths
