"""The evaluator's fixed-point distances where their form changes: a pair of
atoms from 1e-6 to 3,000 A apart (FP64 below 1/4 A, a shift a power of two from
32 A on), around the limits of the fixed-point range (atoms 512 A from the
rotation centre, reference and moved centre 768 A from the origin, coordinates
of 3,000 A), with an i-RMSD partner of its own or the same one.  Tolerance 1e-12
as in the other evaluator tests."""
import numpy as np
import pytest

import gdock_gb300 as gd
from conftest import make_mol, tatom
from test_gpu_evaluator import check

pytestmark = pytest.mark.gpu


def run(oracle, rec, lig, ref, genes):
    got = gd.Evaluator(gd.Complex(rec, lig, []), ref).eval_metrics(genes)
    check(got, oracle.Evaluator(rec, ref).eval_metrics(lig, genes))


@pytest.mark.parametrize("n", [1, 3000])
@pytest.mark.parametrize("far", [1e-6, 0.2, 0.2499999, 0.25, 0.2500001, 1.0, 3.9999, 15.9, 31.999, 32.0, 63.9, 64.1, 500.0, 3000.0])
def test_lengths(oracle, far, n):
    rng = np.random.default_rng(int(far * 1000) + n)
    rec = make_mol([tatom(*rng.normal(0, 2, 3), resseq=1 + k // 4, chain="A") for k in range(12)])
    xyz = rng.normal(0, 3, (9, 3)) + [6.0, 0, 0]
    lig = make_mol([tatom(*x, resseq=1 + k // 3, chain="B", serial=50 + k) for k, x in enumerate(xyz)])
    u = rng.normal(size=(9, 3))
    u *= far / np.linalg.norm(u, axis=1)[:, None]
    ref = make_mol([tatom(*x, resseq=1 + k // 3, chain="B", serial=50 + k) for k, x in enumerate(xyz + u)])
    genes = np.zeros((n, 6))
    genes[1:] = rng.normal(0, 1e-3, (n - 1, 6))
    got = gd.Evaluator(gd.Complex(rec, lig, []), ref).eval_metrics(genes)
    check(got[:20], oracle.Evaluator(rec, ref).eval_metrics(lig, genes[:20]))


@pytest.mark.parametrize("arm", [3.0, 511.9, 512.1, 700.0])
@pytest.mark.parametrize("at", [0.0, 600.0, 767.0, 769.0, 2990.0, 3010.0, 9000.0])
def test_range(oracle, arm, at):
    # two ligand atoms `arm` from their centre, everything `at` along x, the
    # reference atoms in another order (an i-RMSD partner of its own)
    rng = np.random.default_rng(int(arm + at))
    rec = make_mol([tatom(at + k, 0.5, 0, resseq=1, chain="A") for k in range(3)])
    lig = make_mol([tatom(at - arm, 1, 2, resseq=1, chain="B"), tatom(at + arm, 1, 2, resseq=2, chain="B"),
                    tatom(at, 1, 2, resseq=3, chain="B")])
    ref = make_mol([tatom(at + arm - 1.5, 1, 2, resseq=2, chain="B"), tatom(at + 2, 1, 2, resseq=3, chain="B"),
                    tatom(at - arm, 3, 2, resseq=1, chain="B")])
    genes = np.concatenate([np.zeros((1, 6)), rng.uniform(0, 6, (4, 6)), [[1, 2, 3, 760.0, 0, 0], [1, 2, 3, 0, -775.0, 0]]])
    run(oracle, rec, lig, ref, genes)
