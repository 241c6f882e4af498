"""The FP64 step's tile follows the grid (4 x 4 to 16 x 16 cells): grids that
take different tiles, with remainders on either side, in both boundary
conditions, against the oracle bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(3, 5), (17, 9), (40, 40), (41, 100), (100, 80), (129, 63), (7, 300), (200, 201)]


@pytest.mark.parametrize("size", SIZES)
def test_periodic_grids(om_lib, oracle, size):
    h = om_lib.Hydro(size, precision=64, gamma=1.4)
    h.init_kh(5)
    h.set_scalar("cfl", 0.4)
    st = h.state()
    h.proceed(3)
    ref, _, dts = oracle.hydro_run(st, 3, cyclic=True, gamma=1.4, cfl=0.4, dtype=np.float64)
    for x, y in zip(h.state(), ref):
        assert np.array_equal(x, y)
    assert np.array_equal(h.dt_history(3), dts)
    h.close()


@pytest.mark.parametrize("size", SIZES)
def test_open_grids(om_lib, oracle, size):
    h = om_lib.Hydro(size, precision=64, gamma=5 / 3, boundary=om_lib.OPEN)
    for name, v in (("extent0", 1.0), ("extent1", 1.0), ("dR0", 1.0 / size[0]),
                    ("dR1", 1.0 / size[1]), ("cfl", 0.4)):
        h.set_scalar(name, v)
    st = oracle.hydro_init_jet(*size, cyclic=False, gamma=5 / 3, dtype=np.float64)
    h.set_state(st)
    h.proceed(3)
    ref, _, dts = oracle.hydro_run(st, 3, cyclic=False, gamma=5 / 3, cfl=0.4, dtype=np.float64)
    for x, y in zip(h.state(), ref):
        assert np.array_equal(x, y)
    assert np.array_equal(h.dt_history(3), dts)
    h.close()
