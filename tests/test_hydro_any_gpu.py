"""The persistent FP32 step on grids whose sides are no multiples of 32 (partial
tiles, where rows are multiples of 4 cells), against the tile kernels bit for
bit, in its forms with one and two groups per CTA and with few CTAs, so that
each walks many tiles; other rows and open grids keep the tile kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(64, 65), (65, 64), (68, 97), (100, 70), (96, 333), (292, 131), (1000, 200), (776, 401)]
FORMS = [dict(tile_x=16), dict(tile_x=16, grid_limit=3), dict(grid_limit=1), dict(grid_limit=2)]


def start(pg, size, boundary, **cfg):
    h = pg.Hydro(size, precision=32, gamma=1.4, boundary=boundary, **cfg)
    if boundary == pg.OPEN:
        for name, v in (("extent0", 1.0), ("extent1", 1.0), ("dR0", 1.0 / size[0]),
                        ("dR1", 1.0 / size[1])):
            h.set_scalar(name, v)
        h.init()
    else:
        h.init_kh(3)
    h.set_scalar("cfl", 0.4)
    return h


@pytest.mark.parametrize("open_", [False, True])
@pytest.mark.parametrize("size", SIZES)
def test_any_size_equals_the_tile_kernel(om_lib, size, open_):
    pg = om_lib
    boundary = pg.OPEN if open_ else pg.CYCLIC
    ref = start(pg, size, boundary, tile_y=32)
    ref.proceed(7)
    want, dts = ref.state(), ref.dt_history(7)
    ref.close()
    for cfg in FORMS:
        h = start(pg, size, boundary, **cfg)
        h.proceed(7)
        assert np.array_equal(h.dt_history(7), dts), cfg
        for x, y in zip(h.state(), want):
            assert np.array_equal(x, y), cfg
        h.close()


@pytest.mark.parametrize("odd", [[], [(131, 70)]])
@pytest.mark.parametrize("cfg", [{}, {"tile_x": 16}, {"grid_limit": 2}])
def test_uneven_ensembles(om_lib, cfg, odd):
    pg = om_lib
    sizes = [(64, 64), (100, 67), (132, 96), (256, 192), (64, 300), (68, 64)] + odd
    e = pg.Ensemble(sizes, precision=32, gamma=1.4, **cfg)
    e.init_kh(7)
    e.step(6)
    for k, s in enumerate(sizes):
        h = pg.Hydro(s, precision=32, gamma=1.4, tile_y=32)
        h.init_kh(7 + k)
        h.set_scalar("cfl", 0.4)
        h.proceed(6)
        for x, y in zip(e.state(k), h.state()):
            assert np.array_equal(x, y), (s, cfg)
        assert e.scalar(k, "time") == h.get_scalar("time")
        h.close()
    e.close()
