"""FP32 grids of more than 16 tiles of 32 x 32 per SM that the persistent kernel
does not take (rows that are no multiples of 4 cells, open grids): their 32 x 24
tiles against the other tile kernels bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1801, 1600), (2050, 1441)])
@pytest.mark.parametrize("open_", [False, True])
def test_large_grids_equal_the_smaller_tiles(om_lib, size, open_):
    pg = om_lib
    got = []
    for cfg in ({}, {"grid_limit": 1} if open_ else {"tile_y": 32}):
        h = pg.Hydro(size, precision=32, gamma=1.4,
                     boundary=pg.OPEN if open_ else pg.CYCLIC, **cfg)
        if open_:
            for name, v in (("extent0", 1.0), ("extent1", 1.0), ("dR0", 1.0 / size[0]),
                            ("dR1", 1.0 / size[1])):
                h.set_scalar(name, v)
            h.init()
        else:
            h.init_kh(3)
        h.set_scalar("cfl", 0.4)
        h.proceed(4)
        got.append((h.state(), h.dt_history(4)))
        h.close()
    for x, y in zip(got[0][0], got[1][0]):
        assert np.array_equal(x, y)
    assert np.array_equal(got[0][1], got[1][1])
