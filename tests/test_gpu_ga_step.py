"""The device GA step at the population sizes where its sorts change form (two
threads per entry up to 256, one up to 512, the bitonic sort beyond) and with
the Hall of Fame short of, at and beyond its room: populations and Hall of Fame
equal the oracle's bit for bit on the same draws (plain FP64 scoring)."""
import numpy as np
import pytest

import gdock_gb300 as gd
from gdock_gb300 import _lib
from test_gpu_ga import hof_list, setup_job

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pop,top_k,cap", [(2, 1, 4), (24, 24, 24), (254, 10, 500), (256, 300, 500), (258, 10, 45),
                                           (512, 10, 500), (514, 40, 130), (1500, 10, 600)])
def test_populations_and_hall_of_fame(oracle, pop, top_k, cap):
    c, lig = setup_job(8, 6, 2, seed=5)
    cfg = _lib.ga_default_cfg(pop_size=pop, max_generations=6, seed=3, early_stopping=0, hof_max_size=cap,
                              hof_top_k=top_k, elitism=min(5, pop))
    res = gd.run_ga([gd.Complex(c.receptor, lig, c.restraint_pairs)], cfg, gd.GD_PREC_F64, use_graph=False,
                    hall_of_fame=True)
    hof = oracle.HallOfFame(max_size=cap, top_k=top_k)
    genes, _, _, _ = oracle.run_ga(c.receptor, lig, c.restraint_pairs, cfg, _lib.ga_draw(cfg, cfg.seed, 6), hof=hof)
    np.testing.assert_array_equal(res.genes[0], genes)
    assert [(g, gen) for g, _, gen in hof_list(res.hall_of_fame[0])] == [(g, gen) for g, _, gen in hof.entries]


def test_angles_that_wrap(oracle):
    """Mutations of several turns: the wrap by subtraction and by fmod."""
    c, lig = setup_job(8, 6, 2, seed=6)
    cfg = _lib.ga_default_cfg(pop_size=64, max_generations=5, seed=4, early_stopping=0, rot_sigma=9.0, mutation_rate=0.7)
    res = gd.run_ga([gd.Complex(c.receptor, lig, c.restraint_pairs)], cfg, gd.GD_PREC_F64, use_graph=False)
    genes, _, _, _ = oracle.run_ga(c.receptor, lig, c.restraint_pairs, cfg, _lib.ga_draw(cfg, cfg.seed, 5))
    np.testing.assert_array_equal(res.genes[0], genes)
