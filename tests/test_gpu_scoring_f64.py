"""The plain FP64 form where its work split can go wrong: sizes around the
32-atom slots, blocks and segments and around the ligand atoms held at once,
launches of one pose to several hundred (clusters of sixteen CTAs down to
one), coordinates that FP32 cannot resolve and poses that are not finite.

Tolerance: 1e-12 relative to max(|E|, 1 kcal/mol), the bound of the other FP64
tests (the terms differ from the oracle's by a few FP64 roundings each); the
same pose gives the same bits in every launch."""
import numpy as np
import pytest

import gdock_gb300 as gd
from gdock_gb300 import synth
from test_gpu_scoring import F64_TOL, _first_atoms, check

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def big():
    return synth.make_complex(60, 300, 8, seed=41)


@pytest.mark.parametrize("nr,nl", [(1, 1), (31, 33), (32, 32), (33, 31), (64, 65), (65, 1023), (97, 1024), (128, 1025),
                                   (300, 2050)])
def test_sizes_and_launches(oracle, big, nr, nl):
    rec, lig = _first_atoms(big.receptor, nr), _first_atoms(big.ligand, nl)
    lig = gd.position_ligand(rec, lig)
    genes = synth.random_genes(np.random.default_rng(nr + nl), 320, max_displacement=9.0)
    cx = gd.Complex(rec, lig, big.restraint_pairs)
    all_of = cx.score_poses(genes)
    check(all_of[:12], oracle.score_poses(rec, lig, big.restraint_pairs, genes[:12]), F64_TOL)
    for n in (1, 2, 11, 40, 170):
        assert cx.score_poses(genes[:n]).tobytes() == all_of[:n].tobytes(), n
    models = np.stack([np.stack(oracle.apply_genes(lig, g), axis=1) for g in genes[:12]])
    assert cx.score_models(models).tobytes() == all_of[:12].tobytes()


@pytest.mark.parametrize("shift,far", [(3000.0, True), (3890.0, False), (3990.0, False), (1.0e5, True), (3.0e9, True)])
def test_far_from_the_origin(oracle, big, shift, far):
    """Coordinates far from zero: on both sides of the 4,000 A up to which the
    distances come from integers, and up to where FP32 cannot tell atoms apart."""
    rec, lig = _first_atoms(big.receptor, 120), _first_atoms(big.ligand, 90)
    rec = rec.with_coords(rec.x + shift, rec.y - shift, rec.z)
    lig = gd.position_ligand(rec, lig)
    genes = synth.random_genes(np.random.default_rng(3), 6, max_displacement=9.0)
    if far:
        genes[3, 3] = 2.0 * shift  # a pose far away widens the others' bands, too
    cx = gd.Complex(rec, lig, [])
    check(cx.score_poses(genes), oracle.score_poses(rec, lig, [], genes), F64_TOL)


def check_nan(e, ref):
    """check(), with the oracle's NaN and infinities where it has them."""
    for k, name in enumerate(("fitness", "vdw", "elec", "desolv", "air", "restraint_penalty")):
        np.testing.assert_allclose(e[name], ref[:, k], rtol=F64_TOL, atol=F64_TOL, err_msg=name)


def test_poses_that_are_not_finite(oracle, big):
    rec, lig = _first_atoms(big.receptor, 120), _first_atoms(big.ligand, 90)
    lig = gd.position_ligand(rec, lig)
    genes = synth.random_genes(np.random.default_rng(4), 6, max_displacement=9.0)
    genes[1, 3], genes[2, 0], genes[4, 4] = np.inf, np.nan, 1.0e300
    cx = gd.Complex(rec, lig, big.restraint_pairs)
    check_nan(cx.score_poses(genes), oracle.score_poses(rec, lig, big.restraint_pairs, genes))


def test_coincident_atoms_and_vanishing_radii(oracle):
    """Atoms on top of each other (a distance of zero has no vdW and no
    Coulomb term but buries) and Rmin/2 of zero (no vdW energy, but the
    reference's 0 / 0 where r^6 underflows)."""
    from conftest import make_mol, tatom
    rec = make_mol([tatom(float(k), 0, 0, "O", charge=0.5, rmin2=0.0 if k % 2 else 1.8, serial=1 + k) for k in range(5)])
    lig = make_mol([tatom(float(k), 0, 0, "N", charge=-0.25, rmin2=0.0 if k < 3 else 2.0, serial=100 + k) for k in range(5)])
    cx = gd.Complex(rec, lig, [])
    xyz = np.stack([lig.xyz(), lig.xyz() + 1.0e-160, lig.xyz() + [0.0, 1.0e-9, 0.0]])
    check_nan(cx.score_models(xyz), oracle.score_models(rec, lig, [], xyz))


@pytest.mark.parametrize("gene", range(6))
def test_one_undefined_gene(oracle, big, gene):
    """A NaN gene and nothing else out of range: that pose has no pair terms,
    the others keep their bits."""
    rec, lig = _first_atoms(big.receptor, 120), _first_atoms(big.ligand, 90)
    lig = gd.position_ligand(rec, lig)
    genes = synth.random_genes(np.random.default_rng(6), 5, max_displacement=5.0)
    cx = gd.Complex(rec, lig, big.restraint_pairs)
    before = cx.score_poses(genes)
    genes[2, gene] = np.nan
    got = cx.score_poses(genes)
    check_nan(got, oracle.score_poses(rec, lig, big.restraint_pairs, genes))
    keep = [0, 1, 3, 4]
    assert got[keep].tobytes() == before[keep].tobytes()


@pytest.mark.parametrize("axis", range(3))
def test_one_undefined_model_coordinate(oracle, big, axis):
    """One NaN coordinate of one atom of a model: the atom's pairs have no
    term, the model's other atoms and the other models theirs."""
    rec, lig = _first_atoms(big.receptor, 120), _first_atoms(big.ligand, 90)
    lig = gd.position_ligand(rec, lig)
    xyz = lig.xyz()[None] + np.random.default_rng(7).normal(0, 3.0, (4, 1, 3))
    xyz[1, 40, axis] = np.nan
    cx = gd.Complex(rec, lig, big.restraint_pairs)
    check_nan(cx.score_models(xyz), oracle.score_models(rec, lig, big.restraint_pairs, xyz))


@pytest.mark.parametrize("far", [3000.0, 3990.0, 4200.0, 1.0e6, 1.0e300, np.inf, np.nan])
def test_a_pose_beside_one_far_away(oracle, big, far):
    """A pose's record does not depend on the call's other poses, however far
    away they are; nor a model's on the other models."""
    rec, lig = _first_atoms(big.receptor, 120), _first_atoms(big.ligand, 90)
    lig = gd.position_ligand(rec, lig)
    genes = synth.random_genes(np.random.default_rng(8), 6, max_displacement=5.0)
    cx = gd.Complex(rec, lig, big.restraint_pairs)
    alone = cx.score_poses(genes)
    beside = np.concatenate([genes, genes[:1]])
    beside[6, 4] = far
    got = cx.score_poses(beside)
    assert got[:6].tobytes() == alone.tobytes()
    check_nan(got, oracle.score_poses(rec, lig, big.restraint_pairs, beside))
    xyz = lig.xyz()[None] + genes[:, None, 3:]
    models = np.concatenate([xyz, xyz[:1]])
    models[6, 7:70, 1] += far  # some of a model's atoms only
    got = cx.score_models(models)
    assert got[:6].tobytes() == cx.score_models(xyz).tobytes()
    check_nan(got, oracle.score_models(rec, lig, big.restraint_pairs, models))


@pytest.mark.parametrize("stated", [0.0, 8.9, 1.0e4, 1.0e300])
def test_the_stated_displacement_does_not_matter(big, stated):
    """gd_score_frames_device in the FP64 form: max_displacement sizes the FP32
    form's guard bands, FP64 energies are the same bits whatever it says."""
    torch = pytest.importorskip("torch")
    from gdock_gb300 import _lib
    rec, lig = _first_atoms(big.receptor, 120), _first_atoms(big.ligand, 90)
    lig = gd.position_ligand(rec, lig)
    genes = synth.random_genes(np.random.default_rng(9), 40, max_displacement=9.0)
    genes[7, 3] = 5000.0
    cx = gd.Complex(rec, lig, big.restraint_pairs)
    want = cx.score_poses(genes)
    frames = torch.from_numpy(_lib.make_frames(genes)).to("cuda")
    out = torch.zeros((len(genes), 6), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    cx.ctx.check(cx.lib.gd_score_frames_device(cx.h, frames.data_ptr(), len(genes), gd.GD_PREC_F64, stated,
                                               out.data_ptr(), None))
    cx.ctx.sync()
    assert out.cpu().numpy().tobytes() == want.tobytes()


@pytest.mark.parametrize("nr,nl,n", [(40, 4096, 2), (40, 4097, 2), (40, 90000, 1), (40, 90000, 3), (5, 120001, 2)])
def test_long_ligands(oracle, big, nr, nl, n):
    """Ligands of any length: past 4,096 atoms their burial counts are held a turn
    at a time, in a variant of the kernel that checks serials and clamps."""
    from conftest import make_mol, tatom
    rng = np.random.default_rng(nl)
    rec = make_mol([tatom(*x, "CNO"[k % 3], charge=0.3, serial=k + 1) for k, x in enumerate(rng.normal(0, 4.0, (nr, 3)))])
    lig = make_mol([tatom(*x, "CNO"[k % 3], charge=0.2, serial=1000 + k, chain="B")
                    for k, x in enumerate(rng.uniform(-30, 30, (nl, 3)))])
    genes = synth.random_genes(rng, n, max_displacement=9.0)
    cx = gd.Complex(rec, lig, [])
    check(cx.score_poses(genes), oracle.score_poses(rec, lig, [], genes), F64_TOL)


def test_a_refused_receptor_leaves_no_error_behind(oracle, big):
    """A receptor whose counts do not fit a CTA's shared memory is refused;
    the next calls are not (a launch's check reads no older error)."""
    from conftest import make_mol, tatom
    xyz = np.random.default_rng(11).uniform(-90, 90, (150000, 3))
    rec = make_mol([tatom(*x, serial=k + 1) for k, x in enumerate(xyz)])
    lig = make_mol([tatom(0, 0, 0, charge=0.2, serial=200000, chain="B")])
    cx = gd.Complex(rec, lig, [])
    with pytest.raises(Exception, match="shared memory"):
        cx.score_poses(np.zeros((1, 6)))
    rec, lig = _first_atoms(big.receptor, 120), _first_atoms(big.ligand, 90)
    lig = gd.position_ligand(rec, lig)
    genes = synth.random_genes(np.random.default_rng(12), 3, max_displacement=5.0)
    ok = gd.Complex(rec, lig, [])
    assert len(ok.pose_contacts(genes)) == 3
    check(ok.score_poses(genes), oracle.score_poses(rec, lig, [], genes), F64_TOL)


@pytest.mark.parametrize("square", [1e-4, 0.01, 0.1, 0.1249, 0.1251])
def test_small_distances(oracle, square):
    """Pairs of narrow atoms 0.01 to 0.4 A apart, where the integers' step of
    2^-56 A^2 is coarser than a double's."""
    from conftest import make_mol, tatom
    rmin = 0.05 * np.sqrt(square)
    rec = make_mol([tatom(50.0, 3.0, 7.0, charge=0.5, epsilon=-4.0, rmin2=rmin)])
    lig = make_mol([tatom(50.0, 3.0, 7.0, charge=0.3, epsilon=-4.0, rmin2=rmin, serial=9, chain="B")])
    xyz = np.tile(np.array([50.0, 3.0, 7.0]), (20, 1, 1))
    u = np.random.default_rng(10).normal(size=(20, 1, 3))
    xyz += u / np.linalg.norm(u, axis=2)[..., None] * np.sqrt(square)
    got = gd.Complex(rec, lig, []).score_models(xyz)["vdw"]
    ref = oracle.score_models(rec, lig, [], xyz)[:, 1]
    # one term: a dozen FP64 roundings of the reference's and of this form's,
    # 6 r times d2's for r^6
    assert np.abs(got / ref - 1.0).max() <= 2.0 ** -49
