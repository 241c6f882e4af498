"""Populations of Life runs beyond the history kept in host memory (4096
generations) mixed with shorter ones in any order, on every route whose kernels
add to the device counters: tiled rows of whole words, packed rows of any
length, the general kernel of an open grid and the one-CTA grid."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RUNS = (4200, 100, 4150, 30, 2, 4200, 4099, 100)


@pytest.mark.parametrize("use_graph", [0, 1])
@pytest.mark.parametrize("size,open_", [((1056, 24), False), ((1050, 24), False),
                                        ((96, 40), False), ((72, 24), True)])
def test_long_and_short_runs(om_lib, oracle, size, open_, use_graph):
    pg = om_lib
    init = oracle.life_bernoulli(size[0], size[1], 11, 0.35, cyclic=not open_)
    life = pg.Life(size, boundary=pg.OPEN if open_ else pg.CYCLIC, use_graph=use_graph)
    rc, rp = oracle.life_run(init, sum(RUNS), cyclic=not open_)
    life.write("cell", init)
    done = 0
    for gens in RUNS:
        life.proceed(gens)
        assert np.array_equal(life.population_history(gens), rp[done:done + gens]), (gens, done)
        done += gens
        assert life.population == rp[done - 1]
    assert np.array_equal(life.read("cell"), rc)
    life.close()
