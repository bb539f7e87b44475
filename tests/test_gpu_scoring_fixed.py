"""The FP32 kernel's fixed-point transform next to the ends of its range (ligand
atoms 512 A from the rotation centre, the moved centre 768 A from the origin,
coordinates of 4,000 A), where FP64 takes over: against the oracle, charges of
one sign so that no sum cancels."""
import numpy as np
import pytest

import gdock_gb300 as gd
from conftest import make_mol, tatom
from test_gpu_scoring import F32_TOL, check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("at", [0.0, 700.0, 3990.0, 4010.0])
@pytest.mark.parametrize("arm", [5.0, 511.5, 512.5])
def test_range(oracle, at, arm):
    rng = np.random.default_rng(int(at + arm))
    rec = [tatom(at + x, y, z, "CNO"[k % 3], charge=0.3, serial=k + 1) for k, (x, y, z) in enumerate(rng.normal(0, 4.0, (70, 3)))]
    lig = [tatom(at + x, y, z, "CNO"[k % 3], charge=0.2, serial=500 + k, chain="B") for k, (x, y, z) in enumerate(rng.normal(0, 4.0, (40, 3)))]
    # two atoms far out on both sides keep the centre where it is
    lig += [tatom(at - arm, 0, 0, charge=0.2, serial=700, chain="B"), tatom(at + arm, 0, 0, charge=0.2, serial=701, chain="B")]
    R, L = make_mol(rec), make_mol(lig)
    genes = np.zeros((8, 6))
    genes[1:5, :3] = rng.uniform(0, 6.28, (4, 3))
    genes[:5, 3:] = rng.normal(0, 2.0, (5, 3))
    genes[5, 3], genes[6, 4], genes[7, 5] = 767.0, 769.0, -5000.0
    e = gd.Complex(R, L, []).score_poses(genes, gd.GD_PREC_F32)
    check(e, oracle.score_poses(R, L, [], genes), F32_TOL)


@pytest.mark.parametrize("far", [5.0e4, 3.0e6, 1.0e8, np.inf])
def test_poses_beside_one_far_away(oracle, far):
    """A pose so far away that the launch's guard bands cover every distance:
    all pairs of the other poses are re-decided, those beyond 16 A not on
    integers."""
    from gdock_gb300 import synth
    c = synth.make_complex(50, 76, 6, seed=1)
    lig = gd.position_ligand(c.receptor, c.ligand)
    genes = synth.quaternion_genes(np.random.default_rng(2), 24, half_box=12.0)
    genes[7, 3] = far
    e = gd.Complex(c.receptor, lig, c.restraint_pairs).score_poses(genes, gd.GD_PREC_F32)
    ref = oracle.score_poses(c.receptor, lig, c.restraint_pairs, genes)
    keep = np.arange(24) != 7
    check(e[keep], ref[keep], F32_TOL)
