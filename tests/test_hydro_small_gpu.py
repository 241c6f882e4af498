"""The default FP32 step on grids too small to fill the GPU (tiles of 16 x 8
and 32 x 16 cells with more threads), against the 32 x 32 tile kernel bit for
bit, with every CFL time step: the three minima that a run's steps rotate
through must serve runs of any length in any order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def start(pg, size, **cfg):
    h = pg.Hydro(size, precision=32, gamma=1.4, **cfg)
    if cfg.get("boundary", 0) == pg.OPEN:
        for name, v in (("extent0", 1.0), ("extent1", 1.0), ("dR0", 1.0 / size[0]),
                        ("dR1", 1.0 / size[1])):
            h.set_scalar(name, v)
        h.init()
    else:
        h.init_kh(3)
    h.set_scalar("cfl", 0.4)
    return h


@pytest.mark.parametrize("size", [(3, 5), (17, 9), (64, 64), (100, 100), (193, 97), (256, 256),
                                  (257, 200), (500, 300), (391, 411), (500, 700), (512, 512)])
def test_small_grids_equal_the_tile_kernel(om_lib, size):
    a, b = start(om_lib, size), start(om_lib, size, tile_y=32)
    for steps in (1, 2, 3, 4, 4, 2, 2, 5, 1, 3):
        a.proceed(steps)
        b.proceed(steps)
        assert np.array_equal(a.dt_history(steps), b.dt_history(steps))
    for x, y in zip(a.state(), b.state()):
        assert np.array_equal(x, y)
    assert a.get_scalar("time") == b.get_scalar("time")
    a.close()
    b.close()


@pytest.mark.parametrize("size", [(40, 30), (250, 130), (500, 300), (640, 480)])
def test_small_open_grids(om_lib, size):
    # one step per call against runs: other slots, other graphs, same bits
    a, b = start(om_lib, size, boundary=om_lib.OPEN), start(om_lib, size, boundary=om_lib.OPEN,
                                                            grid_limit=1)
    for steps in (1, 2, 4, 4, 3, 5):
        a.proceed(steps)
        for _ in range(steps):
            b.proceed(1)
    for x, y in zip(a.state(), b.state()):
        assert np.array_equal(x, y)
    a.close()
    b.close()


@pytest.mark.parametrize("precision,variant", [(64, 0), (32, 2)])
def test_exact_builds_rotate_too(om_lib, oracle, precision, variant):
    h = om_lib.Hydro((48, 40), precision=precision, variant=variant, gamma=1.4)
    h.init_kh(5)
    h.set_scalar("cfl", 0.4)
    st = h.state()
    total = 0
    for steps in (2, 2, 1, 3, 2, 4):
        h.proceed(steps)
        total += steps
    ref, _, _ = oracle.hydro_run(st, total, cyclic=True, gamma=1.4, cfl=0.4,
                                 dtype=np.float64 if precision == 64 else np.float32)
    for x, y in zip(h.state(), ref):
        assert np.array_equal(x, y)
    h.close()
