"""A run that is repeated is captured from its second time on and replayed from
the fourth at the latest: six equal runs on every route of the dispatch, each
pass compared bit for bit with a machine that captures nothing."""
import numpy as np
import pytest

from paraiso_gb300 import omgraph as og
from paraiso_gb300 import omgraph_examples as ex

pytestmark = pytest.mark.gpu

RUNS = 6


def check_replayed(a, b, replays=3):
    assert a.replay_count() >= replays and b.replay_count() == 0
    a.close()
    b.close()


# one CTA, tiles of whole words, packed tiles, ragged rows, packed with
# warp-specialised ends, the general kernel
@pytest.mark.parametrize("size,gens,open_", [
    ((96, 40), 9, False), ((1536, 200), 20, False), ((1536, 200), 35, False),
    ((1500, 30), 35, False), ((1500, 30), 2, False), ((10240, 3000), 40, False),
    ((100, 70), 3, True), ((100, 70), 4, True)])
def test_life(om_lib, size, gens, open_):
    pg = om_lib
    a, b = [pg.Life(size, boundary=pg.OPEN if open_ else pg.CYCLIC, use_graph=g) for g in (1, 0)]
    for m in (a, b):
        m.fill_random(5, 0.35)
    for _ in range(RUNS):
        for m in (a, b):
            m.proceed(gens)
        assert np.array_equal(a.population_history(gens), b.population_history(gens))
        assert np.array_equal(a.read("cell"), b.read("cell"))
    assert a.generation == RUNS * gens
    check_replayed(a, b)


# the thin tiles, the persistent kernel on whole and partial tiles, 32 x 32 and
# 32 x 24 tiles, open grids, FP64; steps that end in either CFL slot
@pytest.mark.parametrize("steps", [3, 4, 5])
@pytest.mark.parametrize("size,precision,open_", [
    ((100, 100), 32, False), ((256, 256), 32, False), ((384, 256), 32, False),
    ((500, 300), 32, False), ((512, 512), 32, False), ((1000, 700), 32, False),
    ((701, 500), 32, False), ((1801, 1600), 32, False), ((250, 130), 32, True),
    ((701, 500), 32, True), ((64, 48), 64, False), ((65, 48), 64, True)])
def test_hydro(om_lib, size, precision, open_, steps):
    pg = om_lib
    a, b = [pg.Hydro(size, precision=precision, gamma=1.4, use_graph=g,
                     boundary=pg.OPEN if open_ else pg.CYCLIC) for g in (1, 0)]
    for m in (a, b):
        if open_:
            for name, v in (("extent0", 1.0), ("extent1", 1.0), ("dR0", 1.0 / size[0]),
                            ("dR1", 1.0 / size[1])):
                m.set_scalar(name, v)
            m.init()
        else:
            m.init_kh(3)
        m.set_scalar("cfl", 0.4)
    for _ in range(RUNS):
        for m in (a, b):
            m.proceed(steps)
        assert np.array_equal(a.dt_history(steps), b.dt_history(steps))
    for x, y in zip(a.state(), b.state()):
        assert np.array_equal(x, y)
    assert a.get_scalar("time") == b.get_scalar("time")
    check_replayed(a, b)


@pytest.mark.parametrize("steps", [3, 4])
@pytest.mark.parametrize("machine,size", [("life", (256, 192)), ("life", (1000, 400)),
                                          ("hydro", (96, 64)), ("hydro", (500, 300))])
def test_graph_machines(om_lib, oracle, machine, size, steps):
    pg = om_lib
    om = ex.life(size) if machine == "life" else ex.hydro(size, 1.4, "cyclic", og.Float)
    a, b = [pg.GraphMachine(om, use_graph=g) for g in (1, 0)]
    for m in (a, b):
        if machine == "life":
            m.write("cell", oracle.life_bernoulli(size[0], size[1], 7, 0.3))
            continue
        for name, v in (("time", 0.0), ("cfl", 0.4), ("extent0", 1.0), ("extent1", 1.0),
                        ("dR0", 1.0 / size[0]), ("dR1", 1.0 / size[1])):
            m.set_scalar(name, v)
        fields = oracle.hydro_init_kh(size[0], size[1], 3, dtype=np.float32)
        for name, v in zip(("density", "velocity0", "velocity1", "pressure"), fields):
            m.write(name, v)
    scalars = ("population", "generation") if machine == "life" else ("time",)
    for _ in range(RUNS):
        for m in (a, b):
            m.run("proceed", steps)
        for name in scalars:
            assert a.get_scalar(name) == b.get_scalar(name)
    for name in a.array_dtypes:
        assert np.array_equal(a.read(name), b.read(name))
    check_replayed(a, b)


def test_runs_of_ever_other_lengths(om_lib):
    # more lengths than the handle remembers as run once, none twice: nothing is
    # captured; then one of them again and again
    pg = om_lib
    a, b = pg.Life((64, 32)), pg.Life((64, 32), use_graph=0)
    for m in (a, b):
        m.fill_random(5, 0.35)
    for n in range(2, 1100):
        a.proceed(n)
        b.proceed(n)
    assert a.replay_count() == 0 and a.population == b.population
    for _ in range(RUNS):
        a.proceed(5)
        b.proceed(5)
    assert np.array_equal(a.read("cell"), b.read("cell"))
    check_replayed(a, b, replays=1)
