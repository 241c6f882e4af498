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


@pytest.mark.parametrize("open_", [False, True])
@pytest.mark.parametrize("size", [(64, 48), (33, 17), (200, 130)])
def test_fp64_hydro_without_the_stage_state(om_lib, oracle, monkeypatch, size, open_):
    pg = om_lib
    gamma = 5 / 3 if open_ else 1.4
    st = (oracle.hydro_init_jet(*size, cyclic=False, gamma=gamma, dtype=np.float64) if open_ else
          oracle.hydro_init_kh(*size, 5, dtype=np.float64))
    ref, _, dts = oracle.hydro_run(st, 15, cyclic=not open_, gamma=gamma, cfl=0.4,
                                   dtype=np.float64)
    for refused in (True, False):
        if refused:  # the four statics, then the stage-1 state
            monkeypatch.setenv("OM_FAIL_ALLOC_AFTER", "4")
        h = pg.Hydro(size, precision=64, gamma=gamma, boundary=pg.OPEN if open_ else pg.CYCLIC)
        monkeypatch.delenv("OM_FAIL_ALLOC_AFTER", raising=False)
        for name, v in (("extent0", 1.0), ("extent1", 1.0), ("dR0", 1.0 / size[0]),
                        ("dR1", 1.0 / size[1]), ("cfl", 0.4)):
            h.set_scalar(name, v)
        h.set_state(st)
        got = []
        for _ in range(5):
            h.proceed(3)
            got += list(h.dt_history(3))
        assert h.last_launch_count() == (3 if refused else 6)
        for x, y in zip(h.state(), ref):
            assert np.array_equal(x, y)
        assert np.array_equal(got, dts)
        h.close()
