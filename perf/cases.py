"""The calls that users of mbd_b200 make, at the sizes they make them.

Every energy case hands host geometries to ``Engine.energy_batch`` (or
``Engine.energy``) and gets host results back, as a program does that walks
through structures: each pass packs, uploads, computes and downloads.  One
engine serves all of a program's calls; the network of the learned mode is
trained once, before the calls that use it.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from mbd_b200 import synthetic
from mbd_b200.engine import Engine

# The ranges: isolated clusters of 12 (a benzene-sized molecule) to 2000
# atoms; batches of up to 256 clusters of 20 to 600 atoms; graphene sheets
# with a vacuum axis; periodic boxes whose supercell Hamiltonian has up to
# about 6200 rows (1, 8 or 27 cells at the default cut-offs); symmetric
# matrices up to 3000 rows (eigenvalues) and 1200 rows (eigenvectors);
# training sets of 50- to 400-atom clusters.
MODES = ("plain", "mixed", "mixed_learned")
BOX_ATOMS = ((40, 76), (196, 256), (1563, 2000))   # 27, 8 and 1 cells


def listed():
    return [
        # one small molecule, the shortest call there is (a step of a conformer search)
        {"name": "molecule_12_plain", "what": "clusters", "atoms": "12", "mode": "plain", "xc": 1},
        # a drug-sized molecule with the tensor-core relay solve; odd sizes everywhere
        {"name": "molecule_61_mixed", "what": "clusters", "atoms": "61", "mode": "mixed", "xc": 2},
        # a nanocluster at the reference precision
        {"name": "cluster_1000_plain", "what": "clusters", "atoms": "1000", "mode": "plain", "xc": 1},
        # a mid-sized cluster whose size is no multiple of any tile, mixed precision
        {"name": "cluster_533_mixed", "what": "clusters", "atoms": "533", "mode": "mixed", "xc": 1},
        # the benchmark's step: three uneven clusters, learned warm start
        {"name": "clusters_500_1000_2000_learned", "what": "clusters", "atoms": "500,1000,2000",
         "mode": "mixed_learned", "xc": 1},
        # a data set of molecules in one call (the benchmark's batched workload)
        {"name": "batch_256_learned", "what": "batch", "count": 256, "least": 20, "most": 600,
         "mode": "mixed_learned", "xc": 1},
        # the same at the reference precision, a few dozen molecules
        {"name": "batch_40_plain", "what": "batch", "count": 40, "least": 20, "most": 300, "mode": "plain", "xc": 1},
        # a periodic sheet with a vacuum axis (the benchmark's sheet workload)
        {"name": "sheet_128_plain", "what": "sheet", "reps": 8, "mode": "plain", "xc": 1},
        # a small periodic box: a 2 x 2 x 2 supercell, many images
        {"name": "box_256_learned", "what": "box", "atoms": 256, "mode": "mixed_learned", "xc": 1},
        # a periodic box of the benchmark's boxes workload: a 1 x 1 x 1 supercell
        {"name": "box_2000_learned", "what": "box", "atoms": 2000, "mode": "mixed_learned", "xc": 1},
        # the eigenvectors of a Hamiltonian (the modes themselves)
        {"name": "eigenvectors_1051", "what": "eigenvectors", "n": 1051},
        # training the warm start's network, the path's backward direction
        {"name": "training_16", "what": "training", "count": 16, "least": 50, "most": 400, "epochs": 2},
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng: random.Random):
    what = rng.choices(("clusters", "batch", "sheet", "box", "eigenvalues", "eigenvectors", "training"),
                       weights=(8, 3, 2, 3, 1, 1, 1))[0]
    xc = rng.choice((1, 1, 2, 3))
    mode = rng.choice(MODES)
    if what == "clusters":
        sizes = [_log_int(rng, 12, 2000) for _ in range(rng.choice((1, 1, 1, 2, 3)))]
        return {"what": what, "atoms": ",".join(map(str, sizes)), "mode": mode, "xc": xc}
    if what == "batch":
        least = _log_int(rng, 12, 60)
        return {"what": what, "count": _log_int(rng, 8, 160), "least": least, "most": _log_int(rng, 2 * least, 500),
                "mode": mode, "xc": xc}
    if what == "sheet":
        return {"what": what, "reps": rng.randint(3, 9), "mode": mode, "xc": xc}
    if what == "box":
        return {"what": what, "atoms": rng.randint(*rng.choice(BOX_ATOMS)), "mode": mode, "xc": xc}
    if what == "eigenvalues":
        return {"what": what, "n": _log_int(rng, 30, 3000)}
    if what == "eigenvectors":
        return {"what": what, "n": _log_int(rng, 30, 1200)}
    return {"what": what, "count": rng.randint(6, 20), "least": 50, "most": rng.randint(100, 400),
            "epochs": rng.randint(1, 3)}


# ---- inputs -----------------------------------------------------------------
def _geometries(case, seed):
    """The case's (geometry, settings) pairs, from the seed alone (a data set's
    sizes from its case, so that every seed's results have one shape)."""
    rng = np.random.default_rng([seed, 77])
    what = case["what"]
    if what == "clusters":
        pairs = [synthetic.cluster(int(n), int(rng.integers(1 << 31))) for n in case["atoms"].split(",")]
    elif what in ("batch", "training"):
        sizes = np.random.default_rng(case["count"]).integers(case["least"], case["most"] + 1, size=case["count"])
        pairs = [synthetic.cluster(int(n), int(rng.integers(1 << 31))) for n in sizes]
    elif what == "sheet":
        geo, st = synthetic.graphene_sheet(case["reps"])
        geo.coords = geo.coords + rng.uniform(-0.04, 0.04, geo.coords.shape)     # thermal displacements
        geo.hirshfeld = rng.uniform(0.73, 0.81, len(geo.names))
        pairs = [(geo, st)]
    else:
        pairs = [synthetic.periodic_box(case["atoms"], int(rng.integers(1 << 31)))]
    for _, st in pairs:
        st.xc = case.get("xc", 1)
    return [p[0] for p in pairs], [p[1] for p in pairs]


def _matrix(case, seed):
    """A symmetric matrix with the spectrum of a coupled-oscillator
    Hamiltonian: squared frequencies on the diagonal, weaker couplings."""
    n = case["n"]
    rng = np.random.default_rng([seed, 78])
    g = rng.standard_normal((n, n)) * (0.1 / math.sqrt(n))
    return np.diag(rng.uniform(0.15, 0.6, n)) + g + g.T


_ENGINES = {}


def _engine(kind: str) -> Engine:
    """The program's engine ("energies", with its network trained where a
    case asks for the learned mode) and, apart from it, one that trains."""
    if kind not in _ENGINES:
        _ENGINES[kind] = Engine()
    return _ENGINES[kind]


def _with_network(engine: Engine) -> Engine:
    if "network" not in _ENGINES:
        geos, sts = _geometries({"what": "training", "count": 24, "least": 50, "most": 300}, 5)
        engine.learned_train(geos, sts, epochs=4, lr=2e-3, seed=1)
        _ENGINES["network"] = True
    return engine


def prepare(case, seed):
    what = case["what"]
    if what in ("eigenvalues", "eigenvectors"):
        return {"what": what, "engine": _engine("energies"), "H": _matrix(case, seed)}
    geos, sts = _geometries(case, seed)
    if what == "training":
        return {"what": what, "engine": _engine("training"), "geos": geos, "sts": sts, "epochs": case["epochs"]}
    engine = _engine("energies")
    if case["mode"] == "mixed_learned":
        _with_network(engine)
    return {"what": what, "engine": engine, "geos": geos, "sts": sts, "mode": case["mode"]}


# ---- one pass ---------------------------------------------------------------
def run(state):
    eng, what = state["engine"], state["what"]
    if what == "eigenvalues":
        return {"eigenvalues": eng.eigvalsh(state["H"])}
    if what == "eigenvectors":
        w, Z = eng.eigh(state["H"])
        return {"eigenvalues": w, "eigenvectors": Z}
    if what == "training":
        loss = eng.learned_train(state["geos"], state["sts"], epochs=state["epochs"], lr=2e-3, seed=3)
        return {"loss": loss, "parameters": eng.learned_params()}
    if len(state["geos"]) == 1:
        res = [eng.energy(state["geos"][0], state["sts"][0], state["mode"])]
    else:
        res = eng.energy_batch(state["geos"], state["sts"], state["mode"])
    return {
        "energy": np.array([r.energy for r in res]),
        "c6_mol": np.array([r.c6_mol for r in res]),
        "nimag": np.array([r.nimag for r in res]),
        "status": np.array([r.status for r in res]),
        "alpha_eff": np.concatenate([r.alpha_eff for r in res]),
        "c6_eff": np.concatenate([r.c6_eff for r in res]),
        "alpha_iw": np.concatenate([r.alpha_iw for r in res], axis=1),
        "mol_pol_eig": np.stack([r.mol_pol_eig for r in res]),
    }


# ---- what a pass cannot do without ------------------------------------------
def _cells(side):
    return math.ceil(25.0 / side - 1e-9)


def _sizes(case):
    """(atoms, supercell cells) of every geometry, on average for a batch."""
    what = case["what"]
    if what == "clusters":
        return [(int(n), 1) for n in case["atoms"].split(",")]
    if what in ("batch", "training"):
        lo, hi, count = case["least"], case["most"], case["count"]
        return [(lo + (hi - lo) * (k + 0.5) / count, 1) for k in range(count)]
    if what == "sheet":
        return [(2 * case["reps"] ** 2, _cells(2.46 * case["reps"]) ** 2)]
    return [(case["atoms"], _cells((case["atoms"] / synthetic.DENSITY) ** (1 / 3)) ** 3)]


def work(case):
    """Operations of the dense method: for each geometry 21 solves of a
    (3N)-row system for three right-hand sides (factorised; the learned mode
    iterates, some 25 passes over each matrix), and the reduction of the
    coupled-oscillator Hamiltonian.  Bytes: inputs and results."""
    if case["what"] in ("eigenvalues", "eigenvectors"):
        n = float(case["n"])
        if case["what"] == "eigenvalues":
            return {"bytes": 4.0 * n * n + 8.0 * n, "flops": 4.0 / 3.0 * n ** 3}
        return {"bytes": 12.0 * n * n + 8.0 * n, "flops": (4.0 / 3.0 + 2.0) * n ** 3}
    fl = by = 0.0
    for atoms, cells in _sizes(case):
        n = 3.0 * atoms
        factor = 21.0 * n ** 3 / 3.0 + 126.0 * n * n
        if case["what"] == "training":
            # labels by the direct solve; about 40 neighbours of 64 features in 3 layers, forward and backward
            fl += factor + case["epochs"] * 21.0 * atoms * 3.0 * 3.0 * (2 * 40 * 64 + 2 * 2 * 64 * 64)
            by += 36.0 * atoms
            continue
        fl += (21.0 * 25.0 * 6.0 * n * n) if case["mode"] == "mixed_learned" else factor
        fl += 4.0 / 3.0 * (n * cells) ** 3
        by += atoms * 8.0 * (4.5 + 2.0 + 21.0)
    return {"bytes": by, "flops": fl}


# ---- the same in plain torch, in 64 bits ------------------------------------
def _f32(v):
    return float(np.float32(v))


_BOHR = 0.52917721
_GRID = [(0.0, 0.0), (0.0392901, 0.0786611), (0.1183580, 0.0796400), (0.1989120, 0.0816475), (0.2820290, 0.0847872),
         (0.3689190, 0.0892294), (0.4610060, 0.0952317), (0.5600270, 0.1031720), (0.6681790, 0.1136050),
         (0.7883360, 0.1273500), (0.9243900, 0.1456520), (1.0817900, 0.1704530), (1.2684900, 0.2049170),
         (1.4966100, 0.2544560), (1.7856300, 0.3289620), (2.1691700, 0.4480920), (2.7106200, 0.6556060),
         (3.5457300, 1.0659600), (5.0273400, 2.0635700), (8.4489600, 5.6851000), (25.451700, 50.955800)]
_FREE = {"H": (4.5, 6.5, 3.1), "C": (12.0, 46.6, 3.59), "N": (7.4, 24.2, 3.34), "O": (5.4, 15.6, 3.19)}


def _images(lattice, counts):
    ax = [torch.arange(-c, c + 1, dtype=torch.float64, device=lattice.device) for c in counts]
    return -(torch.cartesian_prod(*ax) @ lattice)


def _pair_sum(d0, shifts, cut, six, chunk):
    """Sum over the shifts of six(d, r) (six components) where 0 < r <= cut."""
    acc = None
    step = max(1, chunk // max(1, d0.shape[0] * d0.shape[1]))
    for s in range(0, shifts.shape[0], step):
        d = d0[None] + shifts[s:s + step, None, None]
        r = d.square().sum(-1).sqrt()
        keep = (r <= cut) & (r > 0.0)
        r = torch.where(keep, r, torch.ones_like(r))
        part = six(d, r, keep)
        acc = part if acc is None else acc + part
    return acc


def _blocks(six):
    """(..., 6, N, N) unique components -> (..., 3N, 3N)."""
    xx, xy, xz, yy, yz, zz = six.unbind(-3)
    b = torch.stack([torch.stack([xx, xy, xz], -1), torch.stack([xy, yy, yz], -1), torch.stack([xz, yz, zz], -1)], -2)
    n = b.shape[-3]
    return b.transpose(-3, -2).reshape(*b.shape[:-4], 3 * n, 3 * n)


def _mirror(a):
    """The matrix whose lower triangle this is."""
    return torch.tril(a) + torch.tril(a, -1).transpose(-1, -2)


def _tensor(d, a, b):
    """Sum over the leading (shift) axis of a d d^T + b I, six components."""
    x, y, z = d.unbind(-1)
    return torch.stack([(a * x * x + b).sum(0), (a * x * y).sum(0), (a * x * z).sum(0),
                        (a * y * y + b).sum(0), (a * y * z).sum(0), (a * z * z + b).sum(0)])


def _exact_one(geo, st, dev):
    t64 = dict(dtype=torch.float64, device=dev)
    beta = _f32({1: 0.83, 2: 0.85, 3: 0.85}[st.xc])
    xyz = torch.tensor(geo.coords / _BOHR, **t64)
    lat = torch.tensor(np.asarray(geo.lattice) / _BOHR, **t64)
    v = torch.tensor(geo.hirshfeld, **t64)
    free = torch.tensor([[_f32(q) for q in _FREE[s]] for s in geo.names], **t64)
    a0, c6, r0 = free.unbind(1)
    N = len(geo.names)
    vac = [bool(q) for q in st.mbd_scs_vacuum_axis]
    norm = [float(q) for q in lat.square().sum(1).sqrt()]

    def count(cut, lengths):
        return [0 if (vac[k] or not geo.n_periodic) else math.ceil((cut / _BOHR) / lengths[k]) for k in range(3)]

    sc = [1 if (vac[k] or not geo.n_periodic) else math.ceil((st.mbd_supercell_cutoff / _BOHR) / norm[k])
          for k in range(3)]
    lat_sl = lat * torch.tensor(sc, **t64)[:, None]
    rvdw = v ** (1.0 / 3.0) * r0
    wp = 4.0 / 3.0 * c6 / (a0 * a0)
    d0 = xyz[:, None] - xyz[None]
    # screening: images whose damping factor is not exactly zero in 64 bits
    shifts = _images(lat, count(st.mbd_scs_dip_cutoff, norm))
    reach = 14.5 * beta * float(rvdw.max())
    span = float((xyz.max(0).values - xyz.min(0).values).norm())
    shifts = shifts[shifts.square().sum(1).sqrt() <= reach + span]
    r12 = rvdw[:, None] + rvdw[None]
    alpha_iw, mol = [], []
    eye = torch.eye(3, **t64)
    for w, _ in _GRID:
        w = _f32(w)
        aw = v * a0 / (1.0 + w * w / (wp * wp))
        sg = (aw / 3.0 * math.sqrt(2.0 / math.pi)) ** (1.0 / 3.0)
        s12 = (sg[:, None] ** 2 + sg[None] ** 2).sqrt()
        s12.fill_diagonal_(0.0)
        s12 = s12 + torch.diag(sg)            # an atom with its own images: its own width

        def short(d, r, keep):
            q = r / s12
            ex = torch.exp(-q * q)
            zl = (torch.erf(q) - math.sqrt(4.0 / math.pi) * q * ex) / r ** 5
            zr = math.sqrt(16.0 / math.pi) * ex / (s12 ** 3 * r * r)
            damp = torch.where(keep, 1.0 - 1.0 / (1.0 + torch.exp(-6.0 * (r / (beta * r12) - 1.0))), 0.0)
            return _tensor(d, (-3.0 * zl + zr) * damp, r * r * zl * damp)

        A = _blocks(_pair_sum(d0, shifts, st.mbd_scs_dip_cutoff / _BOHR, short, 12_000_000))
        A = _mirror(A) + torch.diag((1.0 / aw).repeat_interleave(3))
        L, info = torch.linalg.cholesky_ex(A)
        if int(info):
            return None
        X = torch.cholesky_solve(eye.repeat(N, 1), L).reshape(N, 3, 3)
        alpha_iw.append(X.diagonal(dim1=1, dim2=2).mean(1))
        mol.append(X.sum(0))
        del A, L
    alpha_iw, mol = torch.stack(alpha_iw), torch.stack(mol)
    alpha = alpha_iw[0]
    if not bool((alpha > 0).all()):
        return None
    up = torch.triu(mol)
    eig = torch.linalg.eigvalsh((up + torch.triu(mol, 1).transpose(1, 2)).cpu())
    wt = torch.tensor([_f32(g) for _, g in _GRID], **t64)
    c6_mol = 0.954929658551372 * float((wt.cpu() * (eig.sum(1) / 3.0) ** 2)[1:].sum())
    c6_eff = 0.954929658551372 * (wt[1:, None] * alpha_iw[1:] ** 2).sum(0)
    # the coupled oscillators of the supercell
    re = r0 * (alpha / a0) ** (1.0 / 3.0)
    om = 4.0 / 3.0 * c6_eff / alpha ** 2
    re12 = re[:, None] + re[None]
    pref = om[:, None] * om[None] * (alpha[:, None] * alpha[None]).sqrt()
    shifts = _images(lat_sl, count(st.mbd_cfdm_dip_cutoff, [norm[k] * sc[k] for k in range(3)]))

    def long(d, r, keep):
        q = torch.where(keep, 1.0 / (1.0 + torch.exp(-6.0 * (r / (beta * re12) - 1.0))) / r ** 5, 0.0)
        return _tensor(d, -3.0 * q, r * r * q)

    cells = [(i, j, k) for k in range(sc[2]) for j in range(sc[1]) for i in range(sc[0])]
    nsl = len(cells)
    H = torch.zeros(N, nsl, 3, N, nsl, 3, **t64)
    for diff in {tuple(p - q for p, q in zip(a, b)) for a in cells for b in cells}:
        off = torch.tensor([float(q) for q in diff], **t64) @ lat
        six = _pair_sum(d0 + off, shifts, st.mbd_cfdm_dip_cutoff / _BOHR, long, 12_000_000) * pref
        b = _blocks(six).reshape(N, 3, N, 3)
        if diff == (0, 0, 0):
            b = b + torch.diag((om * om).repeat_interleave(3)).reshape(N, 3, N, 3)
        for ra, a in enumerate(cells):
            c = tuple(p - q for p, q in zip(a, diff))
            if c in cells:
                H[:, ra, :, :, cells.index(c), :] = b
    H = _mirror(H.reshape(3 * N * nsl, 3 * N * nsl))
    ev = torch.linalg.eigvalsh(H)
    pos = ev[ev >= 0]
    energy = 0.5 * float(pos.sqrt().sum()) / nsl - 0.5 * float(3.0 * om.sum())
    return {"energy": energy, "c6_mol": c6_mol, "nimag": int((ev < 0).sum()), "alpha_eff": alpha.cpu().numpy(),
            "c6_eff": c6_eff.cpu().numpy(), "alpha_iw": alpha_iw.cpu().numpy(), "mol_pol_eig": eig.numpy()}


def exact(case, seed):
    what = case["what"]
    if what == "eigenvalues":
        return {"eigenvalues": np.linalg.eigvalsh(_matrix(case, seed))}
    if what == "eigenvectors":
        return {"eigenvalues": np.linalg.eigvalsh(_matrix(case, seed)), "eigenvectors": None}   # up to their signs
    if what == "training" or (what == "batch" and case["count"] > 100):
        return None                                                                            # too long here
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    geos, sts = _geometries(case, seed)
    res = [_exact_one(g, s, dev) for g, s in zip(geos, sts)]
    if any(r is None for r in res):
        return None
    return {
        "energy": np.array([r["energy"] for r in res]),
        "c6_mol": np.array([r["c6_mol"] for r in res]),
        "nimag": np.array([r["nimag"] for r in res]),
        "status": np.zeros(len(res), dtype=np.int64),
        "alpha_eff": np.concatenate([r["alpha_eff"] for r in res]),
        "c6_eff": np.concatenate([r["c6_eff"] for r in res]),
        "alpha_iw": np.concatenate([r["alpha_iw"] for r in res], axis=1),
        "mol_pol_eig": np.stack([r["mol_pol_eig"] for r in res]),
    }
