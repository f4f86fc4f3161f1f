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
