"""Clustering where its kernels change form: pose counts around the FCC tiles
and the greedy pass's one CTA or cluster of CTAs, ratios exactly at the
cutoffs, residues of more atoms than a half warp, a warp or the staging takes,
and poses with more contacts than their lists first have room for.  Contacts
and clusters equal the oracle's exactly."""
import numpy as np
import pytest

import gdock_gb300 as gd
from conftest import make_mol, tatom

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 16, 17, 33, 512, 513, 886, 887, 1024, 1025, 1300])
@pytest.mark.parametrize("min_size", [1, 4])
def test_pose_counts(oracle, n, min_size):
    """Sets of 5 to 40 contacts around a few prototypes: many pairs at exactly
    60 % and 45 % common contacts, large clusters and singletons."""
    rng = np.random.default_rng(n)
    protos = [rng.choice(300, 20, replace=False) for _ in range(5)]
    sets = []
    for k in range(n):
        p = protos[k % 5]
        common = p[: int(rng.choice([20, 15, 12, 9, 6]))] if k % 7 else rng.choice(300, int(rng.integers(0, 20)), replace=False)
        sets.append(np.unique(np.concatenate([common, rng.integers(300, 400, int(rng.choice([0, 5, 8])))])).astype(np.int64))
    cfg = gd.ClusteringConfig(min_cluster_size=min_size)
    assert [(r.center_idx, r.members) for r in gd.cluster_sets(sets, cfg)] == oracle.cluster(sets, min_size=min_size)


def residues(rng, sizes, chain, centre):
    atoms = []
    for k, m in enumerate(sizes):
        at = centre + rng.normal(0.0, 5.0, 3)
        atoms += [tatom(*(at + rng.normal(0.0, 1.5, 3)), "C", resseq=k + 1, serial=len(atoms) + 1, chain=chain)
                  for _ in range(m)]
    return make_mol(atoms)


@pytest.mark.parametrize("rec,lig", [([16, 17, 1, 40, 8] * 7, [8, 16, 17, 33] * 4), ([5] * 40, [64, 64, 64, 3, 64]),
                                     ([20] * 9, [65, 4, 4]), ([7], [9])])
def test_large_residues(oracle, rec, lig):
    rng = np.random.default_rng(len(rec))
    R, L = residues(rng, rec, "A", np.zeros(3)), residues(rng, lig, "B", np.zeros(3))
    genes = np.concatenate([rng.uniform(0, 6.28, (24, 3)), rng.normal(0, 7.0, (24, 3))], axis=1)
    cx = gd.Complex(R, L, [])
    sets = [oracle.pose_contacts(R, L, g) for g in genes]
    for a, b in zip(cx.pose_contacts(genes), sets):
        np.testing.assert_array_equal(a, b)
    got = cx.cluster(genes, gd.ClusteringConfig(min_cluster_size=1))
    assert [(r.center_idx, r.members) for r in got] == oracle.cluster(sets, min_size=1)


def test_more_contacts_than_room(oracle):
    """Every residue of one molecule against every one of the other: 6,400
    contacts a pose."""
    rng = np.random.default_rng(1)
    R, L = residues(rng, [1] * 80, "A", np.zeros(3)), residues(rng, [1] * 80, "B", np.zeros(3))
    R, L = (m.with_coords(m.x * 0.1, m.y * 0.1, m.z * 0.1) for m in (R, L))
    genes = np.concatenate([rng.uniform(0, 6.28, (40, 3)), rng.normal(0, 0.5, (40, 3))], axis=1)
    genes[30:, 3] += 4.0
    cx = gd.Complex(R, L, [])
    sets = [oracle.pose_contacts(R, L, g) for g in genes]
    assert max(len(s) for s in sets) > 2048
    for a, b in zip(cx.pose_contacts(genes), sets):
        np.testing.assert_array_equal(a, b)
    assert [(r.center_idx, r.members) for r in cx.cluster(genes)] == oracle.cluster(sets)


def test_lists_within_a_budget():
    """2,000 poses whose lists of 2,048 entries would take 16 MB, with 7 MB left
    in the context's budget: shorter lists, or a bit per residue pair, or half
    of the poses at a time, the same clusters and contacts."""
    from gdock_gb300 import synth
    c = synth.make_complex(50, 76, 0, seed=5)
    lig = gd.position_ligand(c.receptor, c.ligand)
    genes = synth.quaternion_genes(np.random.default_rng(3), 2000, half_box=12.0)
    out = []
    for budget in (0, 1):
        ctx = gd.Context(0)
        cx = gd.Complex(c.receptor, lig, [], ctx=ctx)
        if budget:
            resident = ctx.bytes_in_use
            cx.close()
            ctx.close()
            ctx = gd.Context(0, hbm_budget_bytes=resident + (7 << 20))
            cx = gd.Complex(c.receptor, lig, [], ctx=ctx)
        try:
            keys = cx.pose_contacts(genes)
            out.append(([(r.center_idx, r.members) for r in cx.cluster(genes)], [k.tobytes() for k in keys]))
        finally:
            cx.close()
            ctx.close()
    assert out[0] == out[1]


def test_beside_scoring_on_a_stream():
    """An FP32 gd_score_frames_device call returns before its launch has run, so
    a clustering call made right after it must not use that launch's memory:
    energies and clusters are those of the calls alone."""
    torch = pytest.importorskip("torch")
    from gdock_gb300 import _lib, synth
    c = synth.make_complex(300, 150, 4, seed=8)
    ctx = gd.Context(0)
    cx = gd.Complex(c.receptor, gd.position_ligand(c.receptor, c.ligand), c.restraint_pairs, ctx=ctx)
    try:
        genes = synth.quaternion_genes(np.random.default_rng(4), 20000, half_box=20.0)
        poses = genes[:3000]  # rows past what small calls keep beside the contact lists
        frames = torch.from_numpy(_lib.make_frames(genes)).to("cuda")
        out = torch.zeros((len(genes), 6), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        stream = torch.cuda.Stream()

        def score():
            ctx.check(ctx.lib.gd_score_frames_device(cx.h, frames.data_ptr(), len(genes), gd.GD_PREC_F32, 20.0,
                                                     out.data_ptr(), stream.cuda_stream))

        def clusters():
            return [(r.center_idx, r.members) for r in cx.cluster(poses, gd.ClusteringConfig(min_cluster_size=1))]

        score()
        stream.synchronize()
        energies, alone = out.cpu().numpy().tobytes(), clusters()
        for _ in range(3):
            out.zero_()
            torch.cuda.synchronize()
            score()
            assert clusters() == alone
            stream.synchronize()
            ctx.sync()
            assert out.cpu().numpy().tobytes() == energies
    finally:
        cx.close()
        ctx.close()


@pytest.mark.parametrize("chains", ["AB", "BA", "AA"])
@pytest.mark.parametrize("rec,lig", [([5] * 40, [4] * 70), ([3] * 300, [3] * 130), ([30], [4] * 64), ([4] * 65, [30])])
def test_order_of_contact_keys(oracle, chains, rec, lig):
    """Keys read off as bits (many contacts for the residue pairs there are) and
    sorted (few), the smaller chain's residues first, numbers from negative on."""
    rng = np.random.default_rng(len(rec) + len(lig))
    R, L = residues(rng, rec, chains[0], np.zeros(3)), residues(rng, lig, chains[1], np.zeros(3))
    R.resseq[:] = R.resseq * 3 - 60
    L.resseq[:] = L.resseq * 5 - 31 + (1 << 13)
    genes = np.concatenate([rng.uniform(0, 6.28, (300, 3)), rng.normal(0, 4.0, (300, 3))], axis=1)
    genes[::3, 3] += 17.0  # a few contacts only
    cx = gd.Complex(R, L, [])
    for n in (7, 300):  # one host thread, several
        for a, b in zip(cx.pose_contacts(genes[:n]), oracle.pose_contacts_many(R, L, genes[:n])):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("n", [3, 200, 886, 887, 1300])
@pytest.mark.parametrize("min_size", [0, 1, 2, 3])
@pytest.mark.parametrize("cutoff,strictness", [(0.6, 0.75), (1.0, 1.0), (0.6, 1.8), (1.1, 1.0)])
def test_clusters_of_one(oracle, n, min_size, cutoff, strictness):
    """Poses with no, few and equal contacts, most alone in their cluster: where
    the greedy pass stops and the rest is numbered on the host.  Cutoffs that no
    ratio meets leave every pose without an edge, its own included."""
    rng = np.random.default_rng(n)
    sets = [np.zeros(0, np.int64) if k % 11 == 3 else np.unique(rng.integers(0, 10 ** 6, int(rng.integers(1, 9)))) for k in range(n)]
    for k in range(0, n - 30, 29):  # pairs, one of three
        sets[k + 17] = sets[k].copy()
        if k % 58 == 0:
            sets[k + 29] = sets[k].copy()
    cfg = gd.ClusteringConfig(fcc_cutoff=cutoff, strictness=strictness, min_cluster_size=min_size)
    want = oracle.cluster(sets, fcc_cutoff=cutoff, strictness=strictness, min_size=min_size)
    assert [(r.center_idx, r.members) for r in gd.cluster_sets(sets, cfg)] == want


@pytest.mark.parametrize("mib", [8, 12, 32])
@pytest.mark.parametrize("backwards", [False, True])
def test_calls_one_after_another_within_a_budget(mib, backwards):
    """What a clustering call keeps does not stand in the way of the calls after
    it, in either order, and contact keys need no second copy of the lists."""
    from gdock_gb300 import synth
    c = synth.make_complex(50, 76, 0, seed=9)
    lig = gd.position_ligand(c.receptor, c.ligand)
    genes = synth.quaternion_genes(np.random.default_rng(3), 3000, half_box=12.0)
    cfg = gd.ga_default_cfg(pop_size=100, max_generations=3, early_stopping=0, seed=1)

    def calls(ctx, cx):
        run = [lambda: cx.score_poses(genes, "f32").tobytes(), lambda: cx.score_poses(genes[:200], "f64").tobytes(),
               lambda: [(r.center_idx, r.members) for r in cx.cluster(genes)],
               lambda: [k.tobytes() for k in cx.pose_contacts(genes)],
               lambda: gd.run_ga([cx], cfg, "f32", ctx=ctx).genes.tobytes(),
               lambda: gd.Complex(c.receptor, lig, [], ctx=ctx).close()]
        out = [f() for f in (run[::-1] if backwards else run)]
        return out[::-1] if backwards else out

    got = []
    for budget in (0, 1):
        ctx = gd.Context(0)
        cx = gd.Complex(c.receptor, lig, [], ctx=ctx)
        if budget:
            resident = ctx.bytes_in_use
            cx.close()
            ctx.close()
            ctx = gd.Context(0, hbm_budget_bytes=resident + (mib << 20))
            cx = gd.Complex(c.receptor, lig, [], ctx=ctx)
        try:
            got.append(calls(ctx, cx))
            assert ctx.lib.gd_last_error(ctx.h) == b""
        finally:
            cx.close()
            ctx.close()
    assert got[0] == got[1]
