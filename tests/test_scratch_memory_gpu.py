"""Runs that would keep extra scratch do without it where it cannot be allocated
(failures injected through OM_FAIL_ALLOC_AFTER), with the same results."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("after", [0, 1])
@pytest.mark.parametrize("size,gens", [((1536, 200), 40), ((1500, 30), 35), ((1500, 30), 2),
                                       ((8192, 700), 70)])
def test_life_without_the_packed_grid(om_lib, oracle, monkeypatch, size, gens, after):
    init = oracle.life_bernoulli(size[0], size[1], 3, 0.35)
    rc, rp = oracle.life_run(init, 5 * gens, cyclic=True)
    life = om_lib.Life(size)
    life.write("cell", init)
    monkeypatch.setenv("OM_FAIL_ALLOC_AFTER", str(after))
    for k in range(5):
        life.proceed(gens)
        assert np.array_equal(life.population_history(gens), rp[k * gens:(k + 1) * gens])
        monkeypatch.delenv("OM_FAIL_ALLOC_AFTER", raising=False)
    assert np.array_equal(life.read("cell"), rc)
    assert life.generation == 5 * gens
    life.close()
