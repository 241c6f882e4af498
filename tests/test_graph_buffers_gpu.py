"""Captured runs and buffers that grow: a run repeated until its graph replays,
then one longer than the kept history (4096 Life generations, 1024 Hydro steps),
whose buffer replaces the one that the graph names, then the first run again.
Every result is compared with a machine that captures nothing."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REPEATS = 7


@pytest.mark.parametrize("size", [(1056, 24), (1050, 24), (96, 40)])
def test_life_runs_around_a_longer_one(om_lib, size):
    pg = om_lib
    a, b = pg.Life(size), pg.Life(size, use_graph=0)
    for m in (a, b):
        m.fill_random(5, 0.35)
    for gens in [40] * REPEATS + [4500] + [40] * REPEATS + [6000, 4500] + [40] * REPEATS:
        for m in (a, b):
            m.proceed(gens)
        assert np.array_equal(a.population_history(gens), b.population_history(gens))
        assert a.population == b.population and a.generation == b.generation
    assert np.array_equal(a.read("cell"), b.read("cell"))
    a.close()
    b.close()


@pytest.mark.parametrize("size,precision", [((100, 100), 32), ((128, 96), 32), ((64, 48), 64)])
def test_hydro_runs_around_a_longer_one(om_lib, size, precision):
    pg = om_lib
    a, b = [pg.Hydro(size, precision=precision, gamma=1.4, use_graph=g) for g in (1, 0)]
    for m in (a, b):
        m.init_kh(3)
        m.set_scalar("cfl", 0.4)
    for steps in [20] * REPEATS + [1100] + [20] * REPEATS + [1300] + [20] * REPEATS:
        for m in (a, b):
            m.proceed(steps)
        assert np.array_equal(a.dt_history(steps), b.dt_history(steps))
        assert a.get_scalar("time") == b.get_scalar("time")
    for x, y in zip(a.state(), b.state()):
        assert np.array_equal(x, y)
    a.close()
    b.close()
