"""Life runs through the packed grid (rows of any length from 33 cells, and
long runs of any grid beyond one CTA) against the oracle: rows that end 1, 31
or 8 cells into a word, tiles that wrap in both axes, grids narrower or lower
than a tile, and run lengths around the launches they are split into."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(pg, oracle, size, gens, seed=3, parts=1):
    init = oracle.life_bernoulli(size[0], size[1], seed, 0.35)
    life = pg.Life(size)
    life.write("cell", init)
    rc, rp = oracle.life_run(init, gens * parts, cyclic=True)
    for k in range(parts):
        life.proceed(gens)
        assert np.array_equal(life.population_history(gens), rp[k * gens:(k + 1) * gens])
    assert np.array_equal(life.read("cell"), rc)
    assert life.population == rp[-1] and life.generation == gens * parts
    life.close()


@pytest.mark.parametrize("gens", [2, 33, 70])
@pytest.mark.parametrize("size", [(33, 64), (63, 5), (65, 9), (95, 300), (1000, 70), (1023, 77),
                                  (961, 1), (1921, 513), (4001, 37), (40, 3000)])
def test_ragged_rows(om_lib, oracle, size, gens):
    check(om_lib, oracle, size, gens)


@pytest.mark.parametrize("size,gens", [((1024, 160), 33), ((2048, 2048), 100), ((992, 3001), 65),
                                       ((32, 5000), 131), ((8192, 17), 40), ((3040, 4096), 57),
                                       ((10240, 3000), 34), ((12032, 4000), 90)])
def test_long_runs(om_lib, oracle, size, gens):
    # packed register blocks, and the warp-specialised ends on the large grids
    check(om_lib, oracle, size, gens)


@pytest.mark.parametrize("gens", [1, 2, 7, 64, 301])
@pytest.mark.parametrize("size", [(1, 1), (1, 9), (3, 3), (31, 2), (32, 1), (33, 40), (80, 48),
                                  (96, 33), (128, 128), (127, 129), (160, 100), (512, 60),
                                  (1000, 8), (1024, 17), (992, 1)])
def test_one_cta_grids(om_lib, oracle, size, gens):
    # rows of 1 to 32 words, lane groups that do not fill the warp, fewer rows
    # than the halo
    check(om_lib, oracle, size, gens)


def test_one_cta_long_run(om_lib, oracle):
    check(om_lib, oracle, (70, 20), 4097)   # more generations than one launch counts


@pytest.mark.parametrize("cfg", [{"life_kernel": 5}, {"depth": 3, "tile_x": 4, "tile_y": 8},
                                 {"life_io": 1}])
def test_knobs_do_not_apply_to_small_grids(om_lib, oracle, cfg):
    init = oracle.life_bernoulli(512, 256, 7, 0.3)
    for gens in (20, 50):
        life = om_lib.Life((512, 256), **cfg)
        life.write("cell", init)
        life.proceed(gens)
        rc, rp = oracle.life_run(init, gens, cyclic=True)
        assert np.array_equal(life.read("cell"), rc)
        assert np.array_equal(life.population_history(gens), rp)
        life.close()


def test_graph_replay_and_parity(om_lib, oracle):
    check(om_lib, oracle, (200, 130), 35, parts=3)
    check(om_lib, oracle, (1536, 200), 35, parts=3)


def test_ragged_nonbinary_first_step(om_lib, oracle):
    init = oracle.life_bernoulli(250, 96, 2, 0.3)
    init[10, 10], init[20, 249], init[50, 0] = 3, -1, 7
    life = om_lib.Life((250, 96))
    life.write("cell", init)
    life.proceed(30)
    rc, rp = oracle.life_run(init, 30, cyclic=True)
    assert np.array_equal(life.read("cell"), rc)
    assert np.array_equal(life.population_history(30), rp)
    life.close()


def test_results_in_host_memory(om_lib, oracle):
    # populations and scalars across runs that keep their history on the host
    # (up to 4096 generations) and on the device, in any order, and host writes
    # to the scalars between runs
    for size in ((96, 40), (1500, 30), (2048, 160)):
        init = oracle.life_bernoulli(size[0], size[1], 4, 0.35)
        life = om_lib.Life(size)
        life.write("cell", init)
        total = 0
        rc, rp = oracle.life_run(init, 4700, cyclic=True)
        for k, gens in enumerate((3, 4100, 2, 2, 500, 7, 7, 7)):
            if k == 4:
                life.generation = 1000
            life.proceed(gens)
            assert np.array_equal(life.population_history(gens), rp[total:total + gens])
            total += gens
            assert life.population == rp[total - 1]
            assert life.generation == (total if k < 4 else total - 4107 + 1000)
        life.init()
        assert life.population == 0 and life.generation == 0
        assert life.population_history(5).size == 0
        life.close()
