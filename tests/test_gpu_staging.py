"""The host side of the scoring and evaluation calls, at the sizes where it
changes: frames read and energies written in pinned memory by the kernel itself
(up to 1,024 poses), inputs staged on one or many host threads, and
inputs beyond the staging buffer.  A pose's record does not depend on the call
it came in, so every call equals its pieces."""
import numpy as np
import pytest

import gdock_gb300 as gd
from gdock_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cx():
    c = synth.make_complex(12, 20, 2, seed=3)
    ctx = gd.Context(0)
    cx = gd.Complex(c.receptor, gd.position_ligand(c.receptor, c.ligand), c.restraint_pairs, ctx=ctx)
    yield cx
    cx.close()
    ctx.close()


@pytest.mark.parametrize("prec", [gd.GD_PREC_F32, gd.GD_PREC_F64])
@pytest.mark.parametrize("n", [1, 33, 1024, 1025])
def test_poses(cx, n, prec):
    genes = synth.quaternion_genes(np.random.default_rng(n), n, half_box=12.0)
    whole = cx.score_poses(genes, prec)
    got = [cx.score_poses(genes[i:i + 700], prec) for i in range(0, n, 700)]
    assert np.concatenate(got).tobytes() == whole.tobytes()


@pytest.mark.parametrize("mib", [0.1, 1.1, 70])
def test_models(cx, mib):
    n = max(2, int(mib * 2 ** 20 / 24 / len(cx.ligand)))
    rng = np.random.default_rng(n)
    xyz = cx.ligand.xyz()[None] + rng.normal(0, 3.0, (n, 1, 3))
    whole = cx.score_models(xyz, gd.GD_PREC_F32)
    at = np.unique(np.concatenate([[0, n - 1], rng.integers(0, n, 9)]))
    # the guard band follows the furthest coordinate of the call: decisions and
    # so the energies do not depend on it
    assert cx.score_models(xyz[at], gd.GD_PREC_F32).tobytes() == whole[at].tobytes()


@pytest.mark.parametrize("n", [1, 4097, 450000])
def test_metrics(cx, n):
    ev = gd.Evaluator(cx, cx.ligand)
    genes = synth.quaternion_genes(np.random.default_rng(n), n, half_box=5.0)
    whole = ev.eval_metrics(genes)
    at = np.unique(np.concatenate([[0, n - 1], np.random.default_rng(1).integers(0, n, 9)]))
    assert ev.eval_metrics(genes[at]).tobytes() == whole[at].tobytes()
