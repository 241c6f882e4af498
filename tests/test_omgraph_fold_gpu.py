"""The executor's fold of per-block reduce partials (one partial per 256 cells
up to eight blocks per SM): counts around the 256 threads that fold them, and
NaN and signed zeros where the sequential fold gives them a meaning."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def machine(pg, n):
    from paraiso_gb300 import omgraph as og
    om = og.OM("Fold", (n,), "cyclic")
    d, i = om.static_array("d", og.Double), om.static_array("i", og.Int)
    out = [om.static_scalar(s, t) for s, t in (("dmin", og.Double), ("dmax", og.Double),
                                               ("dsum", og.Double), ("isum", og.Int),
                                               ("imin", og.Int), ("imax", og.Int))]
    k = om.kernel("fold")
    dv, iv = k.load(d), k.load(i)
    for s, (op, v) in zip(out, (("min", dv), ("max", dv), ("sum", dv), ("sum", iv), ("min", iv),
                                ("max", iv))):
        k.store(s, k.reduce(op, v))
    return pg.GraphMachine(om)


@pytest.mark.parametrize("cells", [1, 256, 257, 255 * 256, 256 * 256 + 1, 257 * 256, 152 * 8 * 256,
                                   152 * 8 * 256 + 77])
def test_fold(om_lib, cells):
    rng = np.random.default_rng(cells)
    d = rng.integers(-1000, 1000, cells).astype(np.float64)  # sums are exact in any order
    i = rng.integers(-2**31, 2**31, cells).astype(np.int32)
    at = cells - 1
    d[at], i[at] = 2000.0, 2**31 - 1
    if cells > 1:
        d[at // 2], i[at // 2] = -2000.0, -2**31
    m = machine(om_lib, cells)
    m.write("d", d.reshape(1, -1))
    m.write("i", i.reshape(1, -1))
    m.run("fold")
    assert m.get_scalar("dmin") == d.min() and m.get_scalar("dmax") == d.max()
    assert m.get_scalar("dsum") == d.sum()
    assert m.get_scalar("isum") == int(i.astype(np.int64).sum().astype(np.int32))
    assert m.get_scalar("imin") == i.min() and m.get_scalar("imax") == i.max()
    if cells > 1:  # a NaN that is not the first value counts for nothing in min and max
        d[at] = np.nan
        m.write("d", d.reshape(1, -1))
        m.run("fold")
        assert m.get_scalar("dmin") == -2000.0 and m.get_scalar("dmax") == np.nanmax(d)
        assert np.isnan(m.get_scalar("dsum"))
    m.close()


def test_fold_keeps_the_first_of_equal_zeros(om_lib):
    cells = 600 * 256
    m = machine(om_lib, cells)
    for first, second in ((0.0, -0.0), (-0.0, 0.0)):
        d = np.ones(cells)
        d[300 * 256], d[550 * 256] = first, second
        m.write("d", d.reshape(1, -1))
        m.run("fold")
        assert np.signbit(m.get_scalar("dmin")) == np.signbit(first)
    m.close()
