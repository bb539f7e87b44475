"""The FP32 kernel's runs of near and far rows at every remainder of its steps
(four rows, two for one or two rows left): k receptor atoms close to one ligand
slot and m at 14 A from it, against the oracle and against every other variant
of the kernel and the 16-pose, split and whole-pose forms, whose energies are
the same bits; and the automatic number of receptor parts."""
import numpy as np
import pytest

import gdock_gb300 as gd
from conftest import make_mol, tatom
from gdock_gb300 import _lib, synth
from test_gpu_scoring import F32_TOL, check

pytestmark = pytest.mark.gpu


# (7, 6): this draw's charges cancel to an electrostatic sum of -2.77, a
# hundredth of its largest terms, so that FP32's rounding of those terms is
# 2.5e-5 of the sum, in this kernel and in its predecessors alike.
CANCELS = pytest.mark.xfail(strict=True, reason="electrostatic terms cancel: 7e-5 absolute is 2.5e-5 of the sum")


@pytest.mark.parametrize("near,far", [pytest.param(n, f, marks=CANCELS if (n, f) == (7, 6) else ())
                                      for n in range(8) for f in (0, 1, 2, 3, 5, 6)])
def test_remainders(oracle, near, far):
    rng = np.random.default_rng(8 * near + far)
    rec = [tatom(*rng.normal(0, 1.5, 3), "CNO"[k % 3], charge=0.3 - 0.1 * k, serial=k + 1) for k in range(near)]
    rec += [tatom(14.5, *rng.normal(0, 0.7, 2), "O", charge=0.4, serial=100 + k) for k in range(far)]
    if not rec:
        rec = [tatom(500.0, 0, 0)]
    lig = [tatom(*rng.normal(0, 1.0, 3), "CNO"[k % 3], charge=0.2 - 0.05 * k, serial=1000 + k, chain="B") for k in range(32)]
    R, L = make_mol(rec), make_mol(lig)
    xyz = np.stack([L.xyz() + rng.normal(0, 0.2, 3) for _ in range(3)])
    ctx = gd.Context(0)
    cx = gd.Complex(R, L, [], ctx=ctx)
    try:
        e = cx.score_models(xyz, gd.GD_PREC_F32)
        check(e, oracle.score_models(R, L, [], xyz), F32_TOL)
        genes = np.zeros((16, 6))
        genes[:, 3:] = rng.normal(0, 0.2, (16, 3))
        pose = cx.score_poses(genes, gd.GD_PREC_F32)
        check(pose, oracle.score_poses(R, L, [], genes), F32_TOL)
        for tune, split in ((324, 1), (68, 1), (324, 2)):
            ctx.set_tuning(_lib.GD_TUNE_F32_SLOTS, tune)
            ctx.set_tuning(_lib.GD_TUNE_SPLIT, split)
            assert cx.score_poses(genes, gd.GD_PREC_F32).tobytes() == pose.tobytes(), (tune, split)
        for tune in (4, 20, 66, 322):  # other step sizes and slots: other orders of the FP32 sums
            ctx.set_tuning(_lib.GD_TUNE_SPLIT, 1)
            ctx.set_tuning(_lib.GD_TUNE_F32_SLOTS, tune)
            check(cx.score_poses(genes, gd.GD_PREC_F32), oracle.score_poses(R, L, [], genes), F32_TOL)
    finally:
        cx.close()
        ctx.close()


@pytest.mark.parametrize("rec,lig,n", [(12, 20, 1), (12, 20, 3000), (300, 60, 1), (300, 60, 150), (300, 60, 1500), (300, 60, 5000)])
def test_automatic_receptor_parts(rec, lig, n):
    """The automatic number of receptor parts (by the launch's items: from 24,
    or one part a segment, down to 1) leaves the energies of whole poses."""
    c = synth.make_complex(rec, lig, 4, seed=rec + n)
    genes = synth.quaternion_genes(np.random.default_rng(n), n, half_box=15.0)
    ctx = gd.Context(0)
    cx = gd.Complex(c.receptor, gd.position_ligand(c.receptor, c.ligand), c.restraint_pairs, ctx=ctx)
    try:
        auto = cx.score_poses(genes, gd.GD_PREC_F32)
        ctx.set_tuning(_lib.GD_TUNE_SPLIT, 1)
        assert cx.score_poses(genes, gd.GD_PREC_F32).tobytes() == auto.tobytes()
    finally:
        cx.close()
        ctx.close()


@pytest.mark.parametrize("rec,lig,n", [(12, 20, 1), (40, 60, 33), (300, 60, 1), (120, 60, 1500)])
def test_shared_serials_in_chunks(oracle, rec, lig, n):
    """Receptor and ligand numbered from 1: the split kernels for equal serials
    give the whole-pose kernel's energies, and the oracle's."""
    c = synth.make_complex(rec, lig, 4, seed=rec + n, overlap_serials=True)
    L = gd.position_ligand(c.receptor, c.ligand)
    genes = synth.quaternion_genes(np.random.default_rng(n), n, half_box=15.0)
    ctx = gd.Context(0)
    cx = gd.Complex(c.receptor, L, c.restraint_pairs, ctx=ctx)
    try:
        auto = cx.score_poses(genes, gd.GD_PREC_F32)
        check(auto[:8], oracle.score_poses(c.receptor, L, c.restraint_pairs, genes[:8]), F32_TOL)
        ctx.set_tuning(_lib.GD_TUNE_SPLIT, 1)
        assert cx.score_poses(genes, gd.GD_PREC_F32).tobytes() == auto.tobytes()
    finally:
        cx.close()
        ctx.close()


def test_seven_near_and_six_far_rows(oracle):
    """7 near and 6 far rows (three left over after a step, two after another)
    with charges of one sign, so that no sum cancels."""
    rng = np.random.default_rng(76)
    rec = [tatom(*rng.normal(0, 1.5, 3), "CNO"[k % 3], charge=0.3, serial=k + 1) for k in range(7)]
    rec += [tatom(14.5, *rng.normal(0, 0.7, 2), "O", charge=0.4, serial=100 + k) for k in range(6)]
    lig = [tatom(*rng.normal(0, 1.0, 3), "CNO"[k % 3], charge=0.2, serial=1000 + k, chain="B") for k in range(32)]
    R, L = make_mol(rec), make_mol(lig)
    xyz = np.stack([L.xyz() + rng.normal(0, 0.2, 3) for _ in range(3)])
    genes = np.zeros((16, 6))
    genes[:, 3:] = rng.normal(0, 0.2, (16, 3))
    ctx = gd.Context(0)
    cx = gd.Complex(R, L, [], ctx=ctx)
    try:
        check(cx.score_models(xyz, gd.GD_PREC_F32), oracle.score_models(R, L, [], xyz), F32_TOL)
        pose = cx.score_poses(genes, gd.GD_PREC_F32)
        check(pose, oracle.score_poses(R, L, [], genes), F32_TOL)
        for tune, split in ((324, 1), (68, 1), (324, 2)):
            ctx.set_tuning(_lib.GD_TUNE_F32_SLOTS, tune)
            ctx.set_tuning(_lib.GD_TUNE_SPLIT, split)
            assert cx.score_poses(genes, gd.GD_PREC_F32).tobytes() == pose.tobytes(), (tune, split)
    finally:
        cx.close()
        ctx.close()
