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


@pytest.mark.parametrize("n", [64, 3000])
def test_near_native_sums_have_no_bias(n):
    """Poses 0.3 to 1 A from the reference structure, the centre at hundreds of
    A: an error that all atoms share does not average out of the RMSD.  Against
    extended precision from the same frames.  Tolerance: centre and displacement
    rounded to 2^-51 A, 8e-16 A on the distance, over 0.25 A and halved by the
    root, and 2.2e-16 for sum, division and root."""
    from gdock_gb300 import _lib
    if np.finfo(np.longdouble).eps > 2e-19:
        pytest.skip("no extended precision here")
    rng = np.random.default_rng(n)
    at = np.array([500.0, -300.0, 200.0])
    rec = make_mol([tatom(*x, resseq=1 + k // 8, chain="A", serial=k + 1)
                    for k, x in enumerate(np.round(at + rng.normal(0, 9, (40, 3)), 3))])
    xyz = np.round(at + rng.normal(0, 8, (300, 3)), 3)
    lig = make_mol([tatom(*x, resseq=1 + k // 8, chain="B", serial=50 + k) for k, x in enumerate(xyz)])
    genes = rng.normal(0, 0.002, (n, 6))
    genes[:, 3:] = rng.uniform(0.25, 0.5, (n, 3)) * rng.choice([-1, 1], (n, 3))
    got = gd.Evaluator(gd.Complex(rec, lig, []), lig).eval_metrics(genes)["rmsd"]
    f = _lib.make_frames(genes).astype(np.longdouble)[:40]  # ca sa cb sb cg sg m01 m02 m11 m12 dx dy dz
    ca, sa, cb, sb, cg, sg, m01, m02, m11, m12 = f[:, :10].T
    rot = np.array([[ca * cb, m01, m02], [sa * cb, m11, m12], [-sb, cb * sg, cb * cg]])  # 3 x 3 x poses
    c = np.array([np.cumsum(v)[-1] / len(v) for v in (lig.x, lig.y, lig.z)]).astype(np.longdouble)
    x = xyz.astype(np.longdouble) - c
    moved = [sum(rot[i, j][:, None] * x[None, :, j] for j in range(3)) + c[i] + f[:, 10 + i, None] for i in range(3)]
    d = np.sqrt(sum((moved[i] - xyz[None, :, i]) ** 2 for i in range(3)))
    assert d.min() > 0.25
    want = np.sqrt(d.sum(axis=1) / len(xyz))
    err = np.abs(got[:40] / want - 1)
    assert err.max() <= 2e-15, float(err.max())
