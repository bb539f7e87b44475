"""The FP64 kernel's search and terms where their forms change: k receptor
atoms near one ligand slot and m farther off, at every remainder of the search's
steps of four rows; pair distances on the ends of the reciprocal's binades; and
terms outside the range of the short sum (charges, well depths and radii many
orders apart).  Charges of one sign, so that no sum cancels; F64_TOL."""
import numpy as np
import pytest

import gdock_gb300 as gd
from conftest import make_mol, tatom
from test_gpu_scoring import F64_TOL, check

pytestmark = pytest.mark.gpu


def run(oracle, rec, lig, xyz=None):
    R, L = make_mol(rec), make_mol(lig)
    x = L.xyz()[None] if xyz is None else xyz
    check(gd.Complex(R, L, []).score_models(x, gd.GD_PREC_F64), oracle.score_models(R, L, [], x), F64_TOL)
    if xyz is None:  # as a rigid pose too: the slot's precomputed sphere
        genes = np.zeros((1, 6))
        check(gd.Complex(R, L, []).score_poses(genes, gd.GD_PREC_F64), oracle.score_poses(R, L, [], genes), F64_TOL)


@pytest.mark.parametrize("near", [0, 1, 2, 3, 4, 5, 31, 32, 33])
@pytest.mark.parametrize("far", [0, 1, 3, 4, 35])
def test_rows(oracle, near, far):
    rng = np.random.default_rng(40 * near + far)
    rec = [tatom(*rng.normal(0, 3.0, 3), "CNO"[k % 3], charge=0.3, serial=k + 1) for k in range(near)]
    rec += [tatom(13.5, *rng.normal(0, 0.7, 2), "O", charge=0.4, serial=100 + k) for k in range(far)]
    rec += [tatom(400.0, 0, 0)]
    lig = [tatom(*rng.normal(0, 1.0, 3), "CNO"[k % 3], charge=0.2, serial=1000 + k, chain="B") for k in range(37)]
    run(oracle, rec, lig)


@pytest.mark.parametrize("square", [2.0, 4.0, 8.0, 16.0, 32.0, 64.5, 128.0, 200.0])
def test_reciprocal_binades(oracle, square):
    # squared distances within some 1e-15 of a power of two, on both sides
    d = np.sqrt(square) * (1.0 + np.arange(-8, 9) * 2.0 ** -52)
    rec = [tatom(0, 0, 0, charge=0.5)]
    lig = [tatom(d[0], 0, 0, charge=0.3, serial=9, chain="B")]
    xyz = np.zeros((len(d), 1, 3))
    xyz[:, 0, 0] = d
    run(oracle, rec, lig, xyz)


@pytest.mark.parametrize("charge", [1.0, 1e-5, 1e-14, 1e-17, 1e-30])
@pytest.mark.parametrize("rmin2", [2.0, 1e-3, 1e-20, 0.7e-50])
def test_terms_far_apart(oracle, charge, rmin2):
    # one pair of usual terms far off, then pairs of small ones alone
    rec = [tatom(0, 0, 0, charge=1.0), tatom(100.0, 0, 0, charge=charge, rmin2=rmin2, epsilon=-0.1 * charge, serial=2)]
    lig = [tatom(0, 3.0, 0, charge=0.5, serial=9, chain="B"), tatom(0, -9.0, 0, charge=0.0, serial=10, chain="B")]
    xyz = np.array([[[0, 3.0, 0], [0, -9.0, 0]], [[100, 3.0, 0], [100, -9.0, 0]], [[100, 11.0, 0], [100, 300.0, 0]]])
    run(oracle, rec, lig, xyz)
