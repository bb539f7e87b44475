"""The DockQ kernel where its forms differ: launches on both sides of the rule
that gives a pose one warp or a CTA, poses on and next to the native one (where
the distances are rounding noise unless the reference's order is kept),
contacts placed around the 5 A cutoff, and poses that are not finite.
Tolerance 1e-12 as in the other evaluator tests; fnat exact."""
import numpy as np
import pytest

import gdock_gb300 as gd
from gdock_gb300 import synth
from test_gpu_evaluator import FIELDS, check

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def case():
    c = synth.make_complex(40, 30, 0, seed=23)
    lig = gd.position_ligand(c.receptor, c.ligand)
    ref = lig.with_coords(lig.x + 12.0, lig.y, lig.z)
    return c.receptor, lig, ref


@pytest.mark.parametrize("n", [1, 33, 2431, 2432, 2433, 5000])
def test_launch_sizes(oracle, case, n):
    rec, lig, ref = case
    genes = synth.random_genes(np.random.default_rng(1), 5000, max_displacement=15.0)[:n]
    ev = gd.Evaluator(gd.Complex(rec, lig, []), ref)
    got = ev.eval_metrics(genes)
    k = min(n, 40)
    check(got[-k:], oracle.Evaluator(rec, ref).eval_metrics(lig, genes[-k:]))
    assert ev.eval_metrics(genes[:k]).tobytes() == got[:k].tobytes()


@pytest.mark.parametrize("step", [0.0, 1.0e-12, 1.0e-6, 0.2, 0.3])
def test_near_the_native_pose(oracle, case, step):
    rec, lig, ref = case
    genes = np.zeros((5, 6))
    genes[:, 3] = 12.0
    genes[1:] += step * np.random.default_rng(2).uniform(-1, 1, size=(4, 6)) * [0.01, 0.01, 0.01, 1, 1, 1]
    got = gd.Evaluator(gd.Complex(rec, lig, []), ref).eval_metrics(genes)
    check(got, oracle.Evaluator(rec, ref).eval_metrics(lig, genes))


def test_contacts_at_the_cutoff(oracle):
    from conftest import make_mol, tatom
    rec = make_mol([tatom(0, 0, 0, resseq=1, chain="A")])
    ref = make_mol([tatom(4.5, 0, 0, resseq=10, chain="B")])
    genes = np.zeros((9, 6))
    genes[:, 3] = 0.5 + np.arange(-4, 5) * 2.0 ** -50
    cx = gd.Complex(rec, ref, [])
    got = gd.Evaluator(cx, ref).eval_metrics(genes)
    check(got, oracle.Evaluator(rec, ref).eval_metrics(ref, genes))
    assert 0.0 < got["fnat"].sum() < 9.0


def test_poses_that_are_not_finite(oracle, case):
    rec, lig, ref = case
    genes = synth.random_genes(np.random.default_rng(3), 6, max_displacement=9.0)
    genes[1, 3], genes[2, 0], genes[4, 4], genes[5, 5] = np.inf, np.nan, 1.0e200, 1.0e20
    got = gd.Evaluator(gd.Complex(rec, lig, []), ref).eval_metrics(genes)
    want = oracle.Evaluator(rec, ref).eval_metrics(lig, genes)
    for k, name in enumerate(FIELDS):
        np.testing.assert_allclose(got[name], want[:, k], rtol=1e-12, atol=1e-300, err_msg=name)
