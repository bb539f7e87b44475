"""The work a docking user has this library do, as cases that can be timed.

Each case is one call (or the short sequence of calls) of a user's program
through the public Python entry points, on seeded synthetic complexes of the
sizes that the repository's tests and benchmark use: receptors of 50 to 2,000
residues, ligands of 20 to 500, 1 to 65,536 poses, both scoring precisions.

``listed()`` gives the fixed cases, ``draw(rng)`` one more from the same
ranges, ``prepare`` what a program holds before the call (the uploaded complex
and the call's inputs), ``run`` one pass, ``work`` what a pass cannot do
without and ``exact`` the same results from plain 64-bit torch and numpy.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import gdock_gb300 as gd
from gdock_gb300 import pdb as gpdb

RESIDUES = ["ALA", "ARG", "ASN", "ASP", "CYS", "GLN", "GLU", "GLY", "HIS", "ILE",
            "LEU", "LYS", "MET", "PHE", "PRO", "SER", "THR", "TRP", "TYR", "VAL"]
ENERGIES = ("fitness", "vdw", "elec", "desolv", "air", "restraint_penalty")
METRICS = ("rmsd", "irmsd", "fnat", "dockq")
ATOMS_PER_RESIDUE = 8.2


def listed():
    return [
        # Chromosome::fitness of one individual, the plain form: the smallest call there is
        dict(name="one_pose_f64", kind="poses", rec=50, lig=76, restraints=6, poses=1, precision="f64", overlap=False),
        # one generation of the reference's population (150) in the plain form, the API's default precision
        dict(name="population_f64", kind="poses", rec=300, lig=150, restraints=12, poses=150, precision="f64",
             overlap=False),
        # a batch of candidate poses rescored in the plain form
        dict(name="batch_f64", kind="poses", rec=300, lig=150, restraints=12, poses=2048, precision="f64",
             overlap=False),
        # one generation of the population in the fast form
        dict(name="population_f32", kind="poses", rec=300, lig=150, restraints=12, poses=150, precision="f32",
             overlap=False),
        # a global scan in the fast form: the benchmark's single-complex workload, the largest scoring call
        dict(name="scan_f32", kind="poses", rec=300, lig=150, restraints=12, poses=65536, precision="f32",
             overlap=False),
        # the `score` command on an ensemble of models; both chains numbered from 1, as in separate PDB files
        dict(name="models_f64", kind="models", rec=173, lig=97, restraints=9, poses=100, precision="f64", overlap=True),
        # a docking run in the plain form, generations and Hall of Fame on the device, then its clusters
        dict(name="dock_f64", kind="dock", rec=50, lig=76, restraints=6, jobs=1, pop=150, generations=25,
             precision="f64", metrics=False),
        # a docking run in the fast form with the per-generation DockQ report
        dict(name="dock_f32", kind="dock", rec=130, lig=90, restraints=8, jobs=1, pop=150, generations=50,
             precision="f32", metrics=True),
        # docking jobs of uneven sizes served together until each converges
        dict(name="serve_f32", kind="serve", rec=300, lig=120, restraints=10, jobs=12, pop=150, generations=60),
        # clusters of a Hall of Fame
        dict(name="cluster_hall", kind="cluster", rec=130, lig=90, restraints=8, poses=183, seeds=8),
        # clusters of a large population of a large complex
        dict(name="cluster_large", kind="cluster", rec=2000, lig=500, restraints=8, poses=4096, seeds=16),
        # DockQ of a large pose set against a known structure
        dict(name="dockq_scan", kind="dockq", rec=300, lig=150, restraints=12, poses=65536),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One case of the listed ranges: sizes over their logarithm, the number
    of poses cut where the call would cost more than the largest listed one."""
    kind = rng.choice(["poses", "poses", "poses", "poses", "models", "dock", "dock", "serve", "cluster", "cluster",
                       "dockq"])
    rec, lig = _log_int(rng, 30, 800), _log_int(rng, 20, 300)
    case = dict(kind=kind, rec=rec, lig=lig, restraints=rng.randint(0, 20))
    pairs = rec * lig
    if kind == "poses":
        case["precision"] = rng.choice(["f64", "f32"])
        # the plain form costs about 140 times the fast one per pose
        most = 2048 * 300 * 150 if case["precision"] == "f64" else 65536 * 300 * 150
        case["poses"] = max(1, min(_log_int(rng, 1, 65536), int(0.9 * most / pairs)))
        case["overlap"] = rng.random() < 0.2
    elif kind == "models":
        case["precision"] = rng.choice(["f64", "f32"])
        case["poses"] = max(1, min(_log_int(rng, 1, 400), int(0.9 * 2048 * 300 * 150 / pairs)))
        case["overlap"] = rng.random() < 0.5
    elif kind == "dock":
        case["precision"] = rng.choice(["f64", "f32", "f32"])
        case["jobs"] = rng.choice([1, 1, 2, 5])
        case["pop"] = 2 * _log_int(rng, 25, 150)
        case["generations"] = _log_int(rng, 5, 60)
        case["metrics"] = rng.random() < 0.4
        most = (2048 if case["precision"] == "f64" else 20000) * 300 * 150
        while case["jobs"] * case["pop"] * (case["generations"] + 1) * pairs > 0.8 * most and case["generations"] > 1:
            case["generations"] -= 1
        if case["jobs"] * case["pop"] * 2 * pairs > 0.8 * most:
            case["jobs"], case["pop"] = 1, 50
    elif kind == "serve":
        case["rec"], case["lig"] = min(rec, 400), min(lig, 150)
        case["jobs"], case["pop"], case["generations"] = rng.randint(2, 12), 150, rng.choice([20, 40, 60])
    elif kind == "cluster":
        case["rec"] = _log_int(rng, 30, 1500)
        case["poses"] = _log_int(rng, 20, 4096)
        case["seeds"] = rng.choice([0, 4, 8, 16])
    else:
        case["poses"] = _log_int(rng, 50, 65536)
    return case


# ------------------------------------------------------------------ inputs --

@functools.lru_cache(maxsize=None)
def _template(resname):
    """Heavy atoms of a residue type, backbone first, with their parameters."""
    names = [a for a in gpdb.residue_atom_names(resname) if not a.startswith("H")]
    back = [a for a in ("N", "CA", "C", "O") if a in names]
    names = back + sorted(a for a in names if a not in back)
    par = [gpdb.type_params(gpdb.atom_type(resname, a)) or {} for a in names]
    return names, [[p.get(k, 0.0) for p in par] for k in ("charge", "epsilon", "rmin2", "eps_1_4", "rmin2_1_4")]


def _radius(n_res):
    return 12.0 * (n_res / 50.0) ** (1.0 / 3.0)


def _chain(rng, n_res, chain, serial0, center):
    """A globular chain at protein density: one residue per cell of a jittered
    lattice in a ball, visited row by row, its other heavy atoms 1.5 to 4 A
    from the C-alpha; coordinates with a PDB file's three decimals."""
    r = _radius(n_res)
    step = (4.0 / 3.0 * math.pi * r ** 3 / n_res) ** (1.0 / 3.0)
    m = int(math.ceil(r / step)) + 1
    ax = np.arange(-m, m + 1) * step
    cells = np.stack(np.meshgrid(ax, ax, ax, indexing="ij"), axis=-1).reshape(-1, 3)
    near = np.argsort(np.linalg.norm(cells, axis=1), kind="stable")[:n_res]
    ca = cells[np.sort(near)] + rng.uniform(-0.8, 0.8, size=(n_res, 3)) + np.asarray(center)
    res = [RESIDUES[k] for k in rng.integers(0, len(RESIDUES), size=n_res)]
    name, resname, idx, par = [], [], [], [[] for _ in range(5)]
    for k, rn in enumerate(res):
        names, p = _template(rn)
        name += names
        resname += [rn] * len(names)
        idx += [k] * len(names)
        for a, b in zip(par, p):
            a += b
    n = len(name)
    off = rng.normal(size=(n, 3))
    off *= (rng.uniform(1.5, 4.0, size=n) / np.linalg.norm(off, axis=1))[:, None]
    off[np.array([a == "CA" for a in name])] = 0.0
    xyz = np.round(ca[np.array(idx)] + off, 3)
    element = [a[0] for a in name]
    radius = {"C": 1.7, "N": 1.55, "O": 1.52}
    return gpdb.Molecule(
        serial=np.arange(serial0, serial0 + n, dtype=np.int32), name=name, altloc=[" "] * n, resname=resname,
        chainid=[chain] * n, resseq=(np.array(idx) + 1).astype(np.int16), icode=[" "] * n,
        x=xyz[:, 0].copy(), y=xyz[:, 1].copy(), z=xyz[:, 2].copy(), occupancy=np.ones(n, np.float32),
        tempfactor=np.zeros(n, np.float32), element=element, charge=np.array(par[0], dtype=np.float64),
        vdw_radius=np.array([radius.get(e, 1.0) for e in element]), epsilon=np.array(par[1], dtype=np.float64),
        rmin2=np.array(par[2], dtype=np.float64), eps_1_4=np.array(par[3], dtype=np.float64),
        rmin2_1_4=np.array(par[4], dtype=np.float64))


def _surface(mol):
    """Residue numbers of the third of the residues farthest from the centre."""
    ca = np.array([i for i, a in enumerate(mol.name) if a == "CA"])
    xyz = mol.xyz()
    d = np.linalg.norm(xyz[ca] - xyz.mean(axis=0), axis=1)
    return mol.resseq[ca[np.argsort(-d, kind="stable")[:max(1, len(ca) // 3)]]]


def _complex(rng, rec, lig, restraints, overlap=False):
    """Receptor, ligand positioned on it, and restraint pairs of surface residues."""
    receptor = _chain(rng, rec, "A", 1, (0.0, 0.0, 0.0))
    ligand = _chain(rng, lig, "B", 1 if overlap else len(receptor) + 1, (_radius(rec) + _radius(lig) + 6.0, 0.0, 0.0))
    rs, ls = _surface(receptor), _surface(ligand)
    k = min(restraints, len(rs), len(ls))
    pairs = [(int(a), int(b)) for a, b in zip(rng.choice(rs, size=k, replace=False), rng.choice(ls, size=k, replace=False))]
    return receptor, gd.position_ligand(receptor, ligand), pairs


def _scan_genes(rng, n, half_box=20.0):
    """Any orientation, centroid in a cube around the receptor's."""
    g = np.empty((n, 6))
    g[:, :3] = rng.uniform(0.0, 2.0 * math.pi, size=(n, 3))
    g[:, 3:] = rng.uniform(-half_box, half_box, size=(n, 3))
    return g


def _docked_genes(rng, n, seeds, contact):
    """Poses touching the receptor's surface, spread around a few placements
    as a converged population is (seeds = 0: every pose a placement of its own)."""
    k = seeds or n
    u = rng.normal(size=(k, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    g = np.concatenate([rng.uniform(0.0, 2.0 * math.pi, size=(k, 3)), u * contact], axis=1)
    if not seeds:
        return g
    g = g[rng.integers(0, seeds, size=n)]
    g[:, :3] = np.mod(g[:, :3] + rng.normal(0.0, 0.05, size=(n, 3)), 2.0 * math.pi)
    g[:, 3:] += rng.normal(0.0, 0.5, size=(n, 3))
    return g


def _ga_cfg(case, **more):
    return gd.ga_default_cfg(pop_size=case["pop"], max_generations=case["generations"], **more)


def _reference(receptor, ligand, rec, lig):
    """The ligand's known placement: touching the receptor along x."""
    d = _radius(rec) + _radius(lig) - 2.0
    return ligand.with_coords(ligand.x + d, ligand.y, ligand.z)


def prepare(case, seed):
    rng = np.random.default_rng([seed, 20260])
    kind = case["kind"]
    if kind == "serve":
        jobs = []
        for j in range(case["jobs"]):
            r = max(30, int(round(case["rec"] * math.exp(rng.uniform(-0.7, 0.7)))))
            l = max(20, int(round(case["lig"] * math.exp(rng.uniform(-0.7, 0.7)))))
            jobs.append(_complex(rng, r, l, case["restraints"]))
        srv = gd.Server(ctx=gd.Context(0), max_slots=64, ga=_ga_cfg(case))
        srv.start()
        return dict(case=case, server=srv, jobs=jobs, seed=seed)
    jobs = [_complex(rng, case["rec"], case["lig"], case["restraints"], case.get("overlap", False))
            for _ in range(case.get("jobs", 1))]
    cxs = [gd.Complex(r, l, p) for r, l, p in jobs]
    state = dict(case=case, complexes=cxs)
    receptor, ligand, _ = jobs[0]
    if kind == "poses":
        state["genes"] = _scan_genes(rng, case["poses"])
    elif kind == "models":
        state["xyz"] = _apply(ligand.xyz(), _scan_genes(rng, case["poses"], 12.0)).numpy()
    elif kind == "cluster":
        state["genes"] = _docked_genes(rng, case["poses"], case["seeds"], _radius(case["rec"]) + _radius(case["lig"]) - 7.0)
    elif kind == "dockq":
        state["evaluator"] = gd.Evaluator(cxs[0], _reference(receptor, ligand, case["rec"], case["lig"]))
        state["genes"] = _scan_genes(rng, case["poses"])
    elif kind == "dock":
        state["cfg"] = _ga_cfg(case, seed=seed, early_stopping=0)
        state["evaluators"] = None
        if case["metrics"]:
            state["evaluators"] = [gd.Evaluator(cx, _reference(r, l, case["rec"], case["lig"]))
                                   for cx, (r, l, _) in zip(cxs, jobs)]
    return state


# --------------------------------------------------------------------- run --

def _energies(e, precision):
    """The record's fields; the fast form's as the single-precision numbers they are."""
    return {k: np.ascontiguousarray(e[k], dtype=np.float64 if precision == "f64" else np.float32) for k in ENERGIES}


def _clusters(result, n):
    """Each pose's cluster by rank (-1: none) and, of the clusters in order, centre and size, filled up to n."""
    rank = np.full(n, -1, np.int64)
    centers, sizes = np.full(n, -1, np.int64), np.zeros(n, np.int64)
    for k, c in enumerate(result):
        rank[c.members] = k
        centers[k], sizes[k] = c.center_idx, c.size
    return dict(rank=rank, centers=centers, sizes=sizes)


def _halls(halls, room):
    """The Hall of Fame entries' genes of every job, filled up to `room`."""
    out = np.full((len(halls), room, 6), np.nan)
    for row, h in zip(out, halls):
        row[:len(h)] = h["genes"]
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "serve":
        srv = state["server"]
        ids = [srv.submit(r, l, p, seed=state["seed"] + j) for j, (r, l, p) in enumerate(state["jobs"])]
        genes, fitness, generations, hall = [], [], [], []
        for i in ids:
            if srv.wait(i) != 2:
                raise RuntimeError("a docking job failed")
            res, g, e, _ = srv.result(i)
            h = srv.hall_of_fame(i)
            srv.release(i)
            genes.append(g)
            fitness.append(np.asarray(e["fitness"], dtype=np.float32))
            generations.append(res.generations)
            hall.append(h)
        return dict(genes=np.stack(genes), fitness=np.stack(fitness), generations=np.array(generations, np.int64),
                    hall=_halls(hall, srv.cfg.ga.hof_max_size))
    cxs = state["complexes"]
    if kind == "poses":
        return _energies(cxs[0].score_poses(state["genes"], case["precision"]), case["precision"])
    if kind == "models":
        return _energies(cxs[0].score_models(state["xyz"], case["precision"]), case["precision"])
    if kind == "cluster":
        return _clusters(cxs[0].cluster(state["genes"]), case["poses"])
    if kind == "dockq":
        m = state["evaluator"].eval_metrics(state["genes"])
        return {k: np.ascontiguousarray(m[k]) for k in METRICS}
    res = gd.run_ga(cxs, state["cfg"], case["precision"], hall_of_fame=True, evaluators=state["evaluators"])
    out = dict(genes=res.genes, fitness=_energies(res.energies, case["precision"])["fitness"], generations=res.generations,
               history=np.asarray(res.history, np.float64 if case["precision"] == "f64" else np.float32),
               hall=_halls(res.hall_of_fame, state["cfg"].hof_max_size))
    for j, (cx, h) in enumerate(zip(cxs, res.hall_of_fame)):
        out["clusters%d" % j] = _clusters(cx.cluster(h["genes"]), state["cfg"].hof_max_size)
    if state["evaluators"]:
        out["dockq"] = np.ascontiguousarray(res.best_metrics["dockq"])
        out["mean_dockq"] = res.mean_dockq
    return out


# -------------------------------------------------------------------- work --

@functools.lru_cache(maxsize=None)
def _within(rec, lig, half_box, reach):
    """Share of the atom pairs within `reach`: two balls of residues, the
    ligand's centre anywhere in the cube (half_box > 0) or in contact."""
    rng = np.random.default_rng(7)
    n = 200000

    def ball(r):
        v = rng.normal(size=(n, 3))
        return v / np.linalg.norm(v, axis=1)[:, None] * (r * rng.random(n) ** (1.0 / 3.0))[:, None]

    if half_box > 0:
        c = rng.uniform(-half_box, half_box, size=(n, 3))
    else:
        c = rng.normal(size=(n, 3))
        c *= ((_radius(rec) + _radius(lig) - 7.0) / np.linalg.norm(c, axis=1))[:, None]
    d = np.linalg.norm(ball(_radius(rec)) - ball(_radius(lig)) - c, axis=1)
    return float(np.mean(d < reach))


def _score_flops(rec, lig, half_box):
    """Operations of one pose's pair terms: distance, Coulomb and test of the
    pairs within 15 A, Lennard-Jones of those within 12 A, counts within 8 A."""
    pairs = rec * lig * ATOMS_PER_RESIDUE ** 2
    return pairs * (12 * _within(rec, lig, half_box, 15.0) + 15 * _within(rec, lig, half_box, 12.0)
                    + 2 * _within(rec, lig, half_box, 8.0)) + 28 * lig * ATOMS_PER_RESIDUE


def work(case):
    kind, rec, lig = case["kind"], case["rec"], case["lig"]
    na, nb = rec * ATOMS_PER_RESIDUE, lig * ATOMS_PER_RESIDUE
    upload = 48 * (na + nb)
    if kind == "poses":
        return dict(bytes=case["poses"] * (48 + 48) + upload, flops=case["poses"] * _score_flops(rec, lig, 20.0))
    if kind == "models":
        return dict(bytes=case["poses"] * (24 * nb + 48) + upload, flops=case["poses"] * _score_flops(rec, lig, 12.0))
    if kind in ("dock", "serve"):
        evals = case["jobs"] * case["pop"] * (case["generations"] + 1)
        return dict(bytes=evals * (48 + 48 + 6 * 16 + 16) + case["jobs"] * upload,
                    flops=evals * _score_flops(rec, lig, 50.0))
    if kind == "cluster":
        # the residue pairs' closest atom pairs (within 5 A) and the pair counts of the contact sets
        near = na * nb * _within(rec, lig, 0.0, 7.0)
        contacts = max(16.0, near / 40.0)
        n = case["poses"]
        return dict(bytes=n * 48 + upload + n * 12, flops=n * (28 * nb + 9 * near) + 0.5 * n * n * contacts / 32)
    return dict(bytes=case["poses"] * (48 + 32) + 32 * 2 * nb, flops=case["poses"] * nb * 40)


# ------------------------------------------------------------------- exact --

def _rotation(genes):
    """Rz(alpha) Ry(beta) Rx(gamma) of each gene vector, n x 3 x 3."""
    a, b, c = (torch.as_tensor(genes[:, k]) for k in range(3))
    ca, sa, cb, sb, cg, sg = a.cos(), a.sin(), b.cos(), b.sin(), c.cos(), c.sin()
    rows = [ca * cb, -sa * cg + ca * sb * sg, sa * sg + ca * sb * cg,
            sa * cb, ca * cg + sa * sb * sg, -ca * sg + sa * sb * cg,
            -sb, cb * sg, cb * cg]
    return torch.stack(rows, dim=1).reshape(-1, 3, 3)


def _apply(xyz, genes):
    """Coordinates rotated about their centroid and moved, n x atoms x 3."""
    x = torch.as_tensor(np.ascontiguousarray(xyz))
    c = x.mean(dim=0)
    return torch.einsum("nij,aj->nai", _rotation(genes), x - c) + c + torch.as_tensor(genes[:, None, 3:])


def _asp(mol):
    """Solvation energy per unit burial of each atom."""
    par = np.array([{"C": 0.012, "S": 0.012, "N": -0.160, "O": -0.160}.get(e, 0.0) for e in mol.element])
    return torch.as_tensor(-par * mol.vdw_radius ** 2 * 4.0 * math.pi)


def _exact_energies(receptor, ligand, pairs, coords):
    """The six energies of each coordinate set, the ligand's n x atoms x 3."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f = lambda v: torch.as_tensor(np.ascontiguousarray(v, dtype=np.float64)).to(dev)  # noqa: E731
    R = f(receptor.xyz())
    eps = torch.sqrt(f(receptor.epsilon)[:, None] * f(ligand.epsilon)[None, :])
    r6 = (f(receptor.rmin2)[:, None] + f(ligand.rmin2)[None, :]) ** 6
    qq = 332.0636 * f(receptor.charge)[:, None] * f(ligand.charge)[None, :]
    differ = torch.as_tensor(receptor.serial[:, None] != ligand.serial[None, :]).to(dev)
    asp_r, asp_l = _asp(receptor).to(dev), _asp(ligand).to(dev)
    ia, ib = [], []
    for a, b in gpdb.restraint_pairs_to_indices(receptor, ligand, pairs):
        ia.append(a)
        ib.append(b)
    step = max(1, int(1.5e8 / (len(receptor) * len(ligand))))
    out = []
    for k in range(0, coords.shape[0], step):
        L = coords[k:k + step].to(dev)
        d2 = (R[None, :, 0, None] - L[:, None, :, 0]) ** 2
        d2 += (R[None, :, 1, None] - L[:, None, :, 1]) ** 2
        d2 += (R[None, :, 2, None] - L[:, None, :, 2]) ** 2
        d = d2.sqrt()
        ratio = r6 / (d2 ** 3 + 0.5 * r6)
        v = (eps * (ratio * ratio - 2.0 * ratio)).clamp(-50.0, 500.0)
        vdw = torch.where((d > 0.0) & (d < 12.0) & differ, v, 0.0).sum(dim=(1, 2))
        del ratio, v
        elec = torch.where((d > 1.0) & (d < 15.0), qq / d2, 0.0).sum(dim=(1, 2))
        near = d < 8.0
        buried = lambda c: (c.to(torch.float64) / 10.0).clamp(max=1.0)  # noqa: E731
        desolv = (buried(near.sum(dim=2)) * asp_r).sum(dim=1) + (buried(near.sum(dim=1)) * asp_l).sum(dim=1)
        if ia:
            r = (R[ia] - L[:, ib]).square().sum(dim=2).sqrt()
            air = (10.0 * (r - 7.0).clamp(min=0.0) ** 2).sum(dim=1)
            penalty = (r > 7.0).sum(dim=1).to(torch.float64)
        else:
            air, penalty = torch.zeros_like(vdw), torch.zeros_like(vdw)
        fitness = 0.4 * vdw + 0.05 * elec + 3.4 * desolv + air
        out.append(torch.stack([fitness, vdw, elec, desolv, air, penalty]).cpu())
    e = torch.cat(out, dim=1).numpy()
    return {k: e[i] for i, k in enumerate(ENERGIES)}


def _exact_metrics(receptor, ligand, reference, genes):
    """DockQ and its parts: interface within 5 A, "RMSD" as the root of the mean distance."""
    R, F = receptor.xyz(), reference.xyz()
    close = np.linalg.norm(R[:, None] - F[None], axis=2) <= 5.0
    rec_if, ref_if = set(receptor.resseq[close.any(axis=1)].tolist()), set(reference.resseq[close.any(axis=0)].tolist())
    rec_i = [i for i, s in enumerate(receptor.resseq.tolist()) if s in rec_if]
    lig_i = [i for i, s in enumerate(ligand.resseq.tolist()) if s in ref_if]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    native, R, F = (torch.as_tensor(np.ascontiguousarray(v)).to(dev) for v in (close[np.ix_(rec_i, lig_i)], R, F))
    out = []
    for k in range(0, len(genes), 1024):
        L = _apply(ligand.xyz(), genes[k:k + 1024]).to(dev)
        dist = torch.linalg.norm(L - F, dim=2)
        rmsd = dist.mean(dim=1).sqrt()
        if lig_i:
            irmsd = dist[:, lig_i].mean(dim=1).sqrt()
            d = torch.linalg.norm(R[rec_i][None, :, None] - L[:, None, lig_i], dim=3)
            fnat = ((d <= 5.0) & native).sum(dim=(1, 2)).to(torch.float64) / int(native.sum())
        else:
            irmsd, fnat = torch.zeros_like(rmsd), torch.zeros_like(rmsd)
        dockq = (fnat + 1.0 / (1.0 + (irmsd / 1.5) ** 2) + 1.0 / (1.0 + (rmsd / 8.5) ** 2)) / 3.0
        out.append(torch.stack([rmsd, irmsd, fnat, dockq]).cpu())
    m = torch.cat(out, dim=1).numpy()
    return {k: m[i] for i, k in enumerate(METRICS)}


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("poses", "models", "dockq"):
        return None  # whole numbers, or a search whose course is its own
    atoms = case["rec"] * case["lig"] * ATOMS_PER_RESIDUE ** 2
    if kind != "dockq" and case["poses"] * atoms > (3e10 if torch.cuda.is_available() else 3e8):
        return None
    rng = np.random.default_rng([seed, 20260])
    receptor, ligand, pairs = _complex(rng, case["rec"], case["lig"], case["restraints"], case.get("overlap", False))
    if kind == "models":
        return _exact_energies(receptor, ligand, pairs, _apply(ligand.xyz(), _scan_genes(rng, case["poses"], 12.0)))
    genes = _scan_genes(rng, case["poses"])
    if kind == "dockq":
        if not torch.cuda.is_available() and case["poses"] > 8192:
            return None
        return _exact_metrics(receptor, ligand, _reference(receptor, ligand, case["rec"], case["lig"]), genes)
    return _exact_energies(receptor, ligand, pairs, _apply(ligand.xyz(), genes))
