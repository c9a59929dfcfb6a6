"""Timed cases of the sparse-GP path, each a call that a program using this
package makes:

  calculator   one structure through SGP_Calculator (a step of ASE MD or of an
               on-the-fly run): per-atom ("local") or SOR uncertainties
  batch        SparseGP.predict_batch on several structures at once, in both
               precisions, equal or ragged sizes, one to three species
  autograd     flare_gb300.autograd.energy and its backward pass
  mapped       MappedPotential (an lmp.flare file) on a batch
  md           flare_gb300.md.Ensemble steps
  train        building a model: training structures and sparse environments
  solve        SparseGP.update_matrices_QR

The weights of a model (sparse set, alpha, L_inv, R_inv) come from plain
numpy, once per model and process, as a program loads its model once and
predicts many structures with it; the structures come from the seed.
``exact`` restates each call in plain FP64 torch and numpy.
"""
import functools
import os
import tempfile
import types

import numpy as np
import torch

import flare_gb300 as fg
from flare_gb300 import _lib, autograd, md
from flare_gb300.calculator import SGP_Calculator
from flare_gb300.mapped import MappedPotential
from flare_gb300.sparse_gp import SGP_Wrapper

SIGMA = 2.0
JITTER = 1e-8
LATTICE = 4.05            # A, the FCC cells
DENSITY = 0.06            # atoms / A^3, the random alloys
DMIN = 1.8
FRACTIONS = {1: (1.0,), 2: (0.5, 0.5), 3: (0.5, 0.3, 0.2)}
NUMBERS = (13, 28, 1)
MASSES = (27.0, 58.0, 1.0)
LJ_FCC = ((0.4,), (2.6,))
LJ_ALLOY = ((0.4, 0.25, 0.1), (1.8, 1.7, 1.5))
LABEL_NOISE = 0.01        # eV per environment energy


# ------------------------------------------------------------- the cases
def listed():
    fcc = dict(system="fcc", species=1, n_max=8, l_max=3, rc=5.0, sparse=200,
               power=2)
    two = dict(system="alloy", species=2, n_max=8, l_max=4, rc=5.5,
               sparse=1000, power=2)
    three = dict(two, species=3)
    return [
        # one ASE MD step of a small cell, the calculator's per-atom stds
        dict(fcc, name="calc_local_fcc32", do="calculator", variance="local",
             atoms=32, sparse=64),
        # the wrapper's default uncertainty on a cell of usual size
        dict(fcc, name="calc_sor_fcc108", do="calculator", variance="SOR",
             atoms=108),
        # one structure of the small FCC model, mixed precision
        dict(fcc, name="batch_fcc256_mixed", do="batch", precision="mixed",
             structures=1, atoms=256, want=15),
        # one 1,000-atom alloy cell in the default precision
        dict(two, name="batch_alloy1000_fp64", do="batch", precision="fp64",
             structures=1, atoms=1000, want=15),
        # the throughput workload: 32 alloy cells of 1,000 atoms
        dict(two, name="batch_alloy1000x32_mixed", do="batch",
             precision="mixed", structures=32, atoms=1000, want=15),
        # a served mix: 3 species, uneven sizes
        dict(three, name="batch_ragged3_mixed", do="batch", precision="mixed",
             structures=12, atoms=0, atoms_min=32, atoms_max=2048, want=15),
        # one large cell, energy, forces and stress only
        dict(fcc, name="batch_fcc97k_mixed", do="batch", precision="mixed",
             structures=1, atoms=97556, want=7, n_max=10, l_max=6,
             sparse=1000),
        # energies inside a torch graph, and their gradient
        dict(two, name="autograd_alloy500x4", do="autograd",
             precision="fp64", structures=4, atoms=500, sparse=500),
        # a mapped (LAMMPS) potential on a batch, its default precision
        dict(two, name="mapped_alloy500x4", do="mapped", precision="fp64",
             structures=4, atoms=500, n_max=6, l_max=3, sparse=300),
        # MD of 8 replicas with the uncertainty check, 10 steps a call
        dict(fcc, name="md_fcc256x8", do="md", precision="mixed",
             structures=8, atoms=256, steps=10),
        # an on-the-fly model from its stored structures: Kuu and Kuf rows
        dict(two, name="train_alloy108x3", do="train", structures=3,
             atoms=108, n_max=6, l_max=3, sparse=24),
        # the solve that follows: 1,200 sparse, 3,900 labels
        dict(name="solve_1200", do="solve", sparse=1200, labels=3900),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    do = rng.choice(["calculator", "batch", "batch", "batch", "autograd",
                     "mapped", "md", "train", "solve"])
    if do == "solve":
        m = _log(rng, 100, 1200)
        return dict(do=do, sparse=m, labels=_log(rng, m, 3900))
    species = rng.choice([1, 1, 2, 2, 3])
    big = species < 3
    c = dict(do=do, system="fcc" if species == 1 else "alloy",
             species=species, n_max=rng.randint(4, 8), l_max=rng.randint(2, 4),
             rc=round(rng.uniform(4.2, 5.5), 2),
             sparse=_log(rng, 20, 1000 if big else 400),
             power=rng.choice([2, 2, 2, 2, 1]))
    if do == "calculator":
        c["variance"] = rng.choice(["local", "SOR"])
        c["sparse"] = _log(rng, 20, 200)
        c["n_max"] = min(c["n_max"], 8 if species == 1 else 5)
        c["atoms"] = _log(rng, 20, 256 if c["variance"] == "local" else 120)
    elif do == "batch":
        c["precision"] = rng.choice(["mixed", "mixed", "fp64"])
        c["want"] = rng.choice([15, 15, 7])
        c["atoms"] = _log(rng, 24, 4000)
        c["structures"] = _log(rng, 1, max(1, min(32, (
            24000 if c["precision"] == "mixed" else 4000) // c["atoms"])))
        if c["structures"] > 2 and rng.random() < 0.5:
            c.update(atoms_min=24, atoms_max=c["atoms"], atoms=0)
    elif do == "autograd":
        c["precision"] = rng.choice(["fp64", "mixed"])
        c["atoms"] = _log(rng, 24, 800)
        c["structures"] = rng.randint(1, 4)
        c["sparse"] = min(c["sparse"], 500)
    elif do == "mapped":
        c["precision"] = rng.choice(["fp64", "mixed"])
        c["n_max"] = min(c["n_max"], 8 if species == 1 else
                         6 if species == 2 else 4)
        c["l_max"] = min(c["l_max"], 3)
        c["atoms"] = _log(rng, 24, 800)
        c["structures"] = rng.randint(1, 6)
        c["sparse"] = min(c["sparse"], 300)
    elif do == "md":
        c.update(system="fcc", species=1, precision="mixed", power=2,
                 atoms=4 * rng.randint(2, 6) ** 3, structures=rng.randint(1, 8),
                 steps=rng.randint(3, 10), sparse=_log(rng, 100, 400),
                 n_max=8, l_max=3, rc=5.0)
    if do == "train":
        c["atoms"] = _log(rng, 20, 120)
        c["structures"] = rng.randint(1, 4)
        c["sparse"] = rng.randint(4, min(30, c["atoms"]))
        c["n_max"] = min(c["n_max"], 8 if species == 1 else 5)
    if c["system"] == "fcc":
        c["sparse"] = min(c["sparse"], 200)
    if c["system"] == "fcc" and c.get("atoms"):
        # whole cubic cells of 4 atoms, at least twice as wide as 4 A
        c["atoms"] = 4 * max(2, round((c["atoms"] / 4) ** (1 / 3))) ** 3
    return c


# ------------------------------------------------- structures, numpy only
def _fcc(atoms, disp, r):
    n = int(round((atoms / 4) ** (1 / 3)))
    basis = np.array([[0, 0, 0], [0, .5, .5], [.5, 0, .5], [.5, .5, 0]])
    g = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"),
                 -1).reshape(-1, 3)
    pos = ((g[:, None, :] + basis[None]) * LATTICE).reshape(-1, 3)
    pos = pos + r.normal(scale=disp, size=pos.shape)
    return np.eye(3) * (LATTICE * n), np.zeros(len(pos), np.int64), pos


def _alloy(atoms, species, r):
    """A disordered alloy in a periodic cube: sites of a cubic grid (as many
    left empty as the grid has too many), each atom anywhere in its share of
    the grid that keeps DMIN to its neighbours."""
    box = (atoms / DENSITY) ** (1 / 3)
    n = int(np.ceil(atoms ** (1 / 3) - 1e-9))
    site = np.sort(r.permutation(n ** 3)[:atoms])
    grid = np.stack(np.unravel_index(site, (n, n, n)), 1)
    free = max(0.05, (box / n - DMIN) / 2)
    pos = grid * (box / n) + r.uniform(-free, free, size=(atoms, 3))
    sp = r.choice(species, size=atoms, p=FRACTIONS[species])
    sp[:species] = np.arange(species)
    return np.eye(3) * box, sp.astype(np.int64), pos


def _structure(case, atoms, r):
    if case["system"] == "fcc":
        # hotter than the training cells, where uncertainties matter; MD
        # starts near the lattice
        hot = case["do"] != "md"
        return _fcc(atoms, r.uniform(0.2, 0.28) if hot else 0.04, r)
    return _alloy(atoms, case["species"], r)


def _inputs(case, seed):
    r = np.random.Generator(np.random.PCG64([11, seed]))
    sizes = [case["atoms"]] * case.get("structures", 1)
    if not case["atoms"]:
        # uneven sizes, spread over the logarithm, in mixed order
        lo, hi = np.log(case["atoms_min"]), np.log(case["atoms_max"])
        sizes = np.exp(lo + (hi - lo) * (np.arange(len(sizes)) * 0.618 % 1))
        sizes = [int(round(x)) for x in sizes]
        if case["system"] == "fcc":
            sizes = [4 * max(2, round((n / 4) ** (1 / 3))) ** 3 for n in sizes]
    return [_structure(case, n, r) for n in sizes]


# ------------------------------------- the path in plain FP64 torch
def _pairs(cell, pos, rc):
    """(i, j, r_ij) of every directed pair of a cubic periodic cell, sorted
    by i.  Minimum images where the cell allows it, else a sweep of images."""
    box = cell[0, 0]
    pos = pos - box * torch.floor(pos / box)
    n = len(pos)
    out = []
    if box >= 2 * rc:
        for a in range(0, n, 2048):
            d = pos[None, :, :] - pos[a:a + 2048, None, :]
            d = d - box * torch.round(d / box)
            i, j = torch.nonzero(((d * d).sum(-1) < rc * rc), as_tuple=True)
            keep = i + a != j
            i, j = i[keep], j[keep]
            out.append((i + a, j, d[i, j]))
        return tuple(torch.cat(x) for x in zip(*out))
    k = int(np.ceil(rc / box))
    for s in np.stack(np.meshgrid(*[np.arange(-k, k + 1)] * 3,
                                  indexing="ij"), -1).reshape(-1, 3):
        d = pos[None, :, :] - pos[:, None, :] + box * torch.as_tensor(
            s, dtype=pos.dtype, device=pos.device)
        r2 = (d * d).sum(-1)
        i, j = torch.nonzero((r2 < rc * rc) & (r2 > 0), as_tuple=True)
        out.append((i, j, d[i, j]))
    i, j, v = (torch.cat(x) for x in zip(*out))
    order = torch.argsort(i, stable=True)
    return i[order], j[order], v[order]


def _harmonics(l_max, u):
    """Orthonormal real spherical harmonics of unit vectors, by the
    recurrence of the associated Legendre functions in z (the powers of x
    and y kept apart); column l^2 + l + m."""
    x, y, z = u[:, 0], u[:, 1], u[:, 2]
    c, s = [torch.ones_like(x)], [torch.zeros_like(x)]
    for m in range(l_max):
        c.append(x * c[m] - y * s[m])
        s.append(x * s[m] + y * c[m])
    out = [None] * (l_max + 1) ** 2
    for m in range(l_max + 1):
        p = [torch.full_like(x, float(np.prod(np.arange(1, 2 * m, 2))))]
        if m < l_max:
            p.append((2 * m + 1) * z * p[0])
        for n in range(m + 2, l_max + 1):
            p.append(((2 * n - 1) * z * p[-1] - (n + m - 1) * p[-2]) / (n - m))
        for n in range(m, l_max + 1):
            f = np.sqrt((2 * n + 1) / (4 * np.pi) *
                        np.prod(1.0 / np.arange(n - m + 1, n + m + 1)))
            if m == 0:
                out[n * n + n] = f * p[n]
            else:
                out[n * n + n + m] = np.sqrt(2) * f * p[n - m] * c[m]
                out[n * n + n - m] = np.sqrt(2) * f * p[n - m] * s[m]
    return torch.stack(out, 1)


def _sum_rows(rows, key, n):
    """Sums of rows with equal keys, in the rows' order on the CPU."""
    out = torch.zeros((n,) + rows.shape[1:], dtype=rows.dtype,
                      device=rows.device)
    return out.index_add(0, key, rows)


def _b2(case, i, j, v, sp):
    """B2 descriptors [N, n_d]: chebyshev basis, quadratic cutoff."""
    n_max, l_max, rc, ns = (case["n_max"], case["l_max"], case["rc"],
                            case["species"])
    r = v.norm(dim=1)
    t = [torch.ones_like(r), r / rc]
    for _ in range(max(0, n_max - 2)):
        t.append(2 * (r / rc) * t[-1] - t[-2])
    g = torch.stack(t[:n_max], 1) * ((rc - r) ** 2)[:, None]
    y = _harmonics(l_max, v / r[:, None])
    n, nh = len(sp), (l_max + 1) ** 2
    a = _sum_rows((g[:, :, None] * y[:, None, :]).reshape(len(r), -1),
                  i * ns + sp[j], n * ns).reshape(n, ns * n_max, nh)
    iu = np.triu_indices(ns * n_max)
    cols = [(a[:, :, q * q:(q + 1) ** 2] @
             a[:, :, q * q:(q + 1) ** 2].transpose(1, 2))[:, iu[0], iu[1]]
            for q in range(l_max + 1)]
    return torch.stack(cols, 2).reshape(n, -1)


def _per_atom_lj(case, i, j, v, sp):
    eps, sig = LJ_FCC if case["system"] == "fcc" else LJ_ALLOY
    eps = torch.tensor(eps, dtype=torch.float64)
    sig = torch.tensor(sig, dtype=torch.float64)
    r = v.norm(dim=1)
    q = (0.5 * (sig[sp[i]] + sig[sp[j]]) / r) ** 6
    return _sum_rows(2 * torch.sqrt(eps[sp[i]] * eps[sp[j]]) * (q * q - q), i,
                     len(sp))


# ----------------------------------------------------------- the weights
def _model_key(case):
    return tuple(case[k] for k in ("system", "species", "n_max", "l_max", "rc",
                                   "sparse", "power"))


def _of_key(key):
    return dict(zip(("system", "species", "n_max", "l_max", "rc", "sparse",
                     "power"), key))


@functools.lru_cache(maxsize=None)
def _weights(key):
    """Per species the sparse descriptors of environments of seeded cells,
    with alpha, L_inv and R_inv of the regularised least-squares fit of the
    environments' Lennard-Jones energies (the QR form of the sparse GP)."""
    case = _of_key(key)
    r = np.random.Generator(np.random.PCG64(77))
    need = int(case["sparse"] * 1.3) + 8
    rows, labels, kinds = [], [], []
    while not kinds or min(np.bincount(
            np.concatenate(kinds), minlength=case["species"])) < need:
        atoms = 256 if case["system"] == "fcc" else 500
        if case["system"] == "fcc":
            cell, sp, pos = _fcc(atoms, 0.05, r)
        else:
            cell, sp, pos = _alloy(atoms, case["species"], r)
        sp = torch.from_numpy(sp)
        i, j, v = _pairs(cell, torch.from_numpy(pos), case["rc"])
        rows.append(_b2(case, i, j, v, sp).numpy())
        labels.append(_per_atom_lj(case, i, j, v, sp).numpy())
        kinds.append(sp.numpy())
    rows, labels, kinds = map(np.concatenate, (rows, labels, kinds))
    out = []
    for s in range(case["species"]):
        at = r.permutation(np.nonzero(kinds == s)[0])[:2 * need]
        d = rows[at] / np.linalg.norm(rows[at], axis=1, keepdims=True)
        m = case["sparse"]
        k = SIGMA ** 2 * (d @ d[:m].T) ** case["power"]
        chol = np.linalg.cholesky(k[:m] + JITTER * np.eye(m))
        q, up = np.linalg.qr(np.vstack([k / LABEL_NOISE, chol.T]))
        b = np.concatenate([labels[at] / LABEL_NOISE, np.zeros(m)])
        up_inv = np.linalg.inv(up)
        out.append((rows[at[:m]], up_inv @ (q.T @ b), np.linalg.inv(chol),
                    up_inv))
    return out


def _block_diag(blocks):
    n = sum(len(b) for b in blocks)
    out = np.zeros((n, n))
    at = 0
    for b in blocks:
        out[at:at + len(b), at:at + len(b)] = b
        at += len(b)
    return out


def _descriptor(case):
    return fg.B2("chebyshev", "quadratic", [0.0, case["rc"]], [],
                 [case["species"], case["n_max"], case["l_max"]])


@functools.lru_cache(maxsize=None)
def _model(key, variance="local"):
    """The program's model: SGP_Wrapper with the weights installed."""
    case = _of_key(key)
    b2 = _descriptor(case)
    w = SGP_Wrapper([fg.NormalizedDotProduct(SIGMA, case["power"])], [b2],
                    case["rc"], 0.1, 0.05, 0.01,
                    {NUMBERS[s]: s for s in range(case["species"])},
                    variance_type=variance)
    weights = _weights(key)
    dv = fg.DescriptorValues()
    dv.n_types, dv.n_descriptors = case["species"], b2.n_descriptors
    dv.descriptors = [d for d, _, _, _ in weights]
    dv.descriptor_norms = [np.linalg.norm(d, axis=1) for d in dv.descriptors]
    dv.n_clusters_by_type = [len(d) for d in dv.descriptors]
    w.sparse_gp.set_weights([fg.ClusterDescriptor.from_values(dv)],
                            np.concatenate([x[1] for x in weights]),
                            _block_diag([x[2] for x in weights]), [b2])
    w.sparse_gp.R_inv = _block_diag([x[3] for x in weights])
    return w


@functools.lru_cache(maxsize=None)
def _potential(key):
    """The model's lmp.flare file, read back as a mapped potential."""
    with tempfile.TemporaryDirectory() as folder:
        name = os.path.join(folder, "lmp.flare")
        _model(key).sparse_gp.write_mapping_coefficients(name, "user", 0)
        return MappedPotential(name)


# ------------------------------------------------------- prepare and run
def prepare(case, seed):
    do = case["do"]
    if do == "solve":
        gp = fg.SparseGP([fg.NormalizedDotProduct(SIGMA, 2)], 0.1, 0.05, 0.01)
        gp.Kuu, gp.Kuf, gp.y, gp.noise_vector = _solve_inputs(case, seed)
        gp.n_labels = case["labels"]
        return dict(do=do, gp=gp)
    items = _inputs(case, seed)
    if do == "train":
        r = np.random.Generator(np.random.PCG64([13, seed]))
        return dict(do=do, case=case, b2=_descriptor(case),
                    items=[x + _labels(x, r, case) for x in items])
    w = _model(_model_key(case), case.get("variance", "local"))
    state = dict(do=do, case=case, gp=w.sparse_gp)
    if do == "calculator":
        cell, sp, pos = items[0]
        state["calc"] = SGP_Calculator(w)
        state["atoms"] = types.SimpleNamespace(
            numbers=np.array(NUMBERS)[sp], cell=cell, positions=pos)
        return state
    if do == "md":
        state["ensemble"] = md.Ensemble(
            w.sparse_gp, w.descriptor_calculators, items, MASSES,
            temperature=100.0, seed=seed, precision=case["precision"])
        return state
    state["structures"] = [
        fg.Structure(cell, sp, pos, case["rc"], w.descriptor_calculators)
        for cell, sp, pos in items]
    if do == "autograd":
        state["positions"] = torch.from_numpy(
            np.concatenate([p for _, _, p in items])).cuda()
        state["positions"].requires_grad_(True)
        state["weight"] = torch.linspace(0.5, 1.5, len(items),
                                         dtype=torch.float64, device="cuda")
    if do == "mapped":
        state["potential"] = _potential(_model_key(case))
    return state


def _labels(item, r, case):
    """Energy and forces of the kind that a training structure carries, and
    the atoms chosen as sparse environments."""
    n = len(item[1])
    return (-3.0 * n + r.normal(), r.normal(scale=0.8, size=(n, 3)),
            sorted(r.choice(n, size=case["sparse"], replace=False).tolist()))


def _solve_inputs(case, seed):
    """Kuu, Kuf, y and noise of one species: kernels of unit rows with a
    decaying spectrum, one energy label in 100 and force labels."""
    r = np.random.Generator(np.random.PCG64([17, seed]))
    m, n, q = case["sparse"], case["labels"], 160
    scale = 1.0 / (1.0 + np.arange(q)) ** 0.5
    x = r.normal(size=(m, q)) * scale + scale
    x /= np.linalg.norm(x, axis=1, keepdims=True)
    z = r.normal(size=(n, q)) * scale
    z -= (z @ x[:, :].mean(0))[:, None] * x.mean(0)
    kuf = 2 * SIGMA ** 2 * (x @ x[r.integers(m, size=n)].T) * (x @ z.T)
    noise = np.full(n, 1 / 0.05 ** 2)
    noise[::100] = 1 / 0.1 ** 2
    y = kuf.T @ r.normal(scale=0.3, size=m) + r.normal(scale=0.05, size=n)
    return SIGMA ** 2 * (x @ x.T) ** 2, kuf, y, noise


def run(state):
    do = state["do"]
    gp = state.get("gp")
    if do == "calculator":
        state["calc"].calculate(state["atoms"])
        return dict(state["calc"].results)
    if do == "batch":
        case = state["case"]
        r = gp.predict_batch(state["structures"], case["want"],
                             case["precision"])
        names = ["energy", "forces", "stress"]
        if case["want"] & _lib.FGB_WANT_LOCAL_VAR:
            names.append("local_var")
        return {k: r[k] for k in names}
    if do == "autograd":
        pos = state["positions"]
        e = autograd.energy(pos, gp, state["structures"],
                            state["case"]["precision"])
        grad, = torch.autograd.grad((e * state["weight"]).sum(), pos)
        return {"energy": e.detach(), "grad": grad}
    if do == "mapped":
        return state["potential"].predict(
            state["structures"], precision=state["case"]["precision"])
    if do == "md":
        ens = state["ensemble"]
        ens.step(state["case"]["steps"], dt=1.0, std_threshold=0.05)
        s = ens.state()
        return {k: s[k] for k in ("positions", "velocities", "forces",
                                  "energy", "kinetic", "flagged")}
    if do == "train":
        gp = fg.SparseGP([fg.NormalizedDotProduct(SIGMA,
                                                  state["case"]["power"])],
                         0.1, 0.05, 0.01)
        for cell, sp, pos, energy, forces, atoms in state["items"]:
            s = fg.Structure(cell, sp, pos, state["case"]["rc"],
                             [state["b2"]])
            s.energy = np.array([energy])
            s.forces = forces.reshape(-1)
            gp.add_training_structure(s)
            gp.add_specific_environments(s, atoms)
        return {"Kuu": gp.Kuu, "Kuf": gp.Kuf, "y": gp.y,
                "noise_vector": gp.noise_vector}
    gp.update_matrices_QR()
    return {"alpha": gp.alpha, "L_inv": gp.L_inv, "R_inv": gp.R_inv}


# ------------------------------------------------------------------ work
def _neighbours(case):
    dens = 4 / LATTICE ** 3 if case["system"] == "fcc" else DENSITY
    return 4 / 3 * np.pi * case["rc"] ** 3 * dens


def work(case):
    do = case["do"]
    if do == "solve":
        m, n = case["sparse"], case["labels"] + case["sparse"]
        # Cholesky, two triangular inverses, the QR and Q^T b
        return {"bytes": 8.0 * (3 * m * m + m * case["labels"] + 2 * n),
                "flops": m ** 3 + 2.0 * n * m * m}
    ns, n_max, nh = case["species"], case["n_max"], (case["l_max"] + 1) ** 2
    nr = ns * n_max
    nd = nr * (nr + 1) // 2 * (case["l_max"] + 1)
    nb = _neighbours(case)
    atoms = (case["atoms"] * case.get("structures", 1) if case["atoms"] else
             case["structures"] * (case["atoms_max"] - case["atoms_min"]) /
             np.log(case["atoms_max"] / case["atoms_min"]))
    m = case["sparse"]
    pair = 2.0 * nb * n_max * nh                   # A of one atom
    b2 = pair + 1.0 * nr * (nr + 1) * nh
    back = 3 * pair + 2.0 * nr * nr * nh           # reverse pass of one atom
    quad = 2.0 * nd * nd if case["power"] == 2 else 2.0 * nd
    if do == "train":
        rows = case["structures"] * m
        cols = case["structures"] * (1 + 3 * case["atoms"])
        return {"bytes": 8.0 * (rows * rows + rows * cols + 3 * atoms),
                "flops": atoms * b2 + rows * atoms / ns * (2.0 * nd + back) +
                rows * rows / ns * 2.0 * nd}
    steps = case.get("steps", 1)
    flops = atoms * (b2 + back)
    weights = 8.0 * ns * m * nd
    if do == "mapped":
        flops += atoms * quad
        weights = 8.0 * ns * (nd * nd if case["power"] == 2 else nd)
    else:
        flops += atoms * 2.0 * m * nd              # k against the sparse set
        flops += atoms * min(quad, 2.0 * m * nd)   # dE/dB2
    var = do in ("md", "calculator") or case.get("want", 7) & 8
    if case.get("variance") == "SOR":
        cols = 1 + 3 * atoms + 6
        flops += atoms * m * back + cols * float(ns * m) ** 2
        weights += 8.0 * ns * m * m
    elif var:
        flops += atoms * float(m) ** 2
        weights += 4.0 * ns * m * m
    io = atoms * (24.0 + 4 + 24 + (8 if var else 0))
    return {"bytes": weights + steps * io, "flops": steps * flops}


# ----------------------------------------------------------------- exact
def _dev(x):
    x = torch.as_tensor(np.ascontiguousarray(x))
    return x.cuda() if torch.cuda.is_available() else x


class _Exact:
    """One structure's descriptors and, by torch's reverse mode through
    them, the gradient of any function of them with respect to the pairs."""

    def __init__(self, case, item):
        cell, sp, pos = item[:3]
        self.n, self.volume = len(sp), abs(np.linalg.det(cell))
        self.sp = _dev(sp)
        self.i, self.j, v = _pairs(cell, _dev(pos), case["rc"])
        self.v = v.requires_grad_(True)
        self.case = case
        self.b2 = _b2(case, self.i, self.j, self.v, self.sp)
        self.unit = self.b2 / self.b2.norm(dim=1, keepdim=True)

    def kernel(self, sparse, s):
        """sigma^2 (d . s)^power of the atoms of one species."""
        at = torch.nonzero(self.sp == s)[:, 0]
        rows = _dev(sparse)
        rows = rows / rows.norm(dim=1, keepdim=True)
        return at, SIGMA ** 2 * (self.unit[at] @ rows.T) ** self.case["power"]

    def efs(self, energy, keep=False):
        """[E, forces 3N, stress 6] of a scalar function."""
        g, = torch.autograd.grad(energy, self.v, retain_graph=keep)
        f = torch.zeros((self.n, 3), dtype=g.dtype, device=g.device)
        f = f.index_add(0, self.i, g).index_add(0, self.j, -g)
        s = -(g.T @ self.v.detach()) / self.volume
        iu = np.triu_indices(3)
        return energy.detach().reshape(1), f, s[iu[0], iu[1]]


def _exact_predict(case, item, var=True):
    x = _Exact(case, item)
    energy = 0.0
    local = torch.zeros(x.n, dtype=torch.float64, device=x.v.device)
    for s, (d, alpha, l_inv, _) in enumerate(_weights(_model_key(case))):
        at, k = x.kernel(d, s)
        energy = energy + (k @ _dev(alpha)).sum()
        if var:
            z = k.detach() @ _dev(l_inv).T
            local[at] = SIGMA ** 2 - (z * z).sum(1)
    return x.efs(energy) + (local,)


def _exact_rows(case, item, rows_by_species):
    """Kernel rows of sparse descriptors against a structure's energy,
    forces and stress, species after species."""
    x = _Exact(case, item)
    out = []
    for s, d in enumerate(rows_by_species):
        if len(d) == 0:
            continue
        _, k = x.kernel(d, s)
        for e in k.sum(0):
            a, f, t = x.efs(e, keep=True)
            out.append(torch.cat([a, f.reshape(-1), t]))
    return torch.stack(out)


def _signed_sqrt(v):
    return np.sign(v) * np.sqrt(np.abs(v))


def _exact_calculator(case, item):
    if case["variance"] == "SOR":
        w = _weights(_model_key(case))
        rows = _exact_rows(case, item, [x[0] for x in w])
        mean = _dev(np.concatenate([x[1] for x in w])) @ rows
        z = rows.T @ _dev(_block_diag([x[3] for x in w]))
        mean, v = mean.cpu().numpy(), (z * z).sum(1).cpu().numpy()
        stds = _signed_sqrt(v[1:-6]).reshape(-1, 3)
    else:
        e, f, t, v = _exact_predict(case, item)
        mean = torch.cat([e, f.reshape(-1), t]).cpu().numpy()
        stds = np.zeros((len(v), 3))
        stds[:, 0] = _signed_sqrt(v.cpu().numpy()) / SIGMA
    s = mean[-6:]
    return {"energy": mean[0], "forces": mean[1:-6].reshape(-1, 3),
            "stress": -s[[0, 3, 5, 4, 2, 1]], "stds": stds}


def _exact_train(case, items):
    ns, m = case["species"], case["sparse"]
    desc = []
    for it in items:
        x = _Exact(case, it)
        by = [[a for a in it[5] if it[1][a] == s] for s in range(ns)]
        desc.append([x.b2.detach()[at].cpu().numpy() for at in by])
    rows = [np.concatenate([d[s] for d in desc]) for s in range(ns)]
    kuu = []
    for d in rows:
        d = d / np.linalg.norm(d, axis=1, keepdims=True)
        kuu.append(SIGMA ** 2 * (d @ d.T) ** case["power"])
    kuf = torch.cat([_exact_rows(case, it, rows)[:, :-6] for it in items], 1)
    y, noise = [], []
    for it in items:
        y += [[it[3]], it[4].reshape(-1)]
        noise += [[1 / 0.1 ** 2], np.full(it[4].size, 1 / 0.05 ** 2)]
    return {"Kuu": _block_diag(kuu), "Kuf": kuf.cpu().numpy(),
            "y": np.concatenate(y), "noise_vector": np.concatenate(noise)}


def _exact_md(case, items, seed):
    mass = torch.full((case["atoms"], 1), MASSES[0], dtype=torch.float64)
    out = {k: [] for k in ("positions", "velocities", "forces", "energy",
                           "kinetic")}
    for q, (cell, sp, pos) in enumerate(items):
        # Maxwell-Boltzmann velocities at 100 K, no net momentum
        r = np.random.Generator(np.random.PCG64(seed + q))
        v = r.normal(size=(len(sp), 3)) * np.sqrt(
            8.617333262e-5 * 100.0 * 9.64853321e-3 / MASSES[0])
        v = torch.from_numpy(v - v.mean(0))
        x = torch.from_numpy(pos)
        e, f, _, _ = _exact_predict(case, (cell, sp, x.numpy()), False)
        for _ in range(case["steps"]):
            v = v + 0.5 * f.cpu() * 9.64853321e-3 / mass
            x = x + v
            e, f, _, _ = _exact_predict(case, (cell, sp, x.numpy()), False)
            v = v + 0.5 * f.cpu() * 9.64853321e-3 / mass
        kin = 0.5 * MASSES[0] * float((v * v).sum()) / 9.64853321e-3
        for k, y in zip(out, (x, v, f.cpu(), e.cpu(), [kin])):
            out[k].append(np.asarray(y))
    return {k: np.concatenate(v) for k, v in out.items()}


def _exact_solve(case, seed):
    kuu, kuf, y, noise = _solve_inputs(case, seed)
    m = len(kuu)
    chol = np.linalg.cholesky(kuu + JITTER * np.eye(m))
    w = np.sqrt(noise)
    q, up = np.linalg.qr(np.vstack([(kuf * w).T, chol.T]))
    sign = np.sign(np.diag(up))
    q, up = q * sign, up * sign[:, None]
    r_inv = np.linalg.inv(up)
    return {"alpha": r_inv @ (q.T @ np.concatenate([w * y, np.zeros(m)])),
            "L_inv": np.linalg.inv(chol), "R_inv": r_inv}


def exact(case, seed):
    do = case["do"]
    if do == "solve":
        return _exact_solve(case, seed)
    items = _inputs(case, seed)
    if do == "train":
        r = np.random.Generator(np.random.PCG64([13, seed]))
        return _exact_train(case, [x + _labels(x, r, case) for x in items])
    if do == "calculator":
        return _exact_calculator(case, items[0])
    if do == "md":
        return _exact_md(case, items, seed)
    got = [_exact_predict(case, it, var=do != "mapped" and
                          case.get("want", 7) & 8) for it in items]
    e = torch.cat([g[0] for g in got])
    f = torch.cat([g[1] for g in got])
    if do == "autograd":
        w = torch.linspace(0.5, 1.5, len(items), dtype=torch.float64)
        n = torch.tensor([len(sp) for _, sp, _ in items])
        return {"energy": e.cpu(),
                "grad": -f.cpu() * w.repeat_interleave(n)[:, None]}
    out = {"energy": e, "forces": f, "stress": torch.stack([g[2] for g in got])}
    if do == "mapped":
        out["atom_energies"] = torch.cat(
            [_exact_atom_energies(case, it) for it in items])
    elif case["want"] & 8:
        out["local_var"] = torch.cat([g[3] for g in got])
    return {k: v.cpu().numpy() for k, v in out.items()}


def _exact_atom_energies(case, item):
    x = _Exact(case, item)
    out = torch.zeros(x.n, dtype=torch.float64, device=x.v.device)
    for s, (d, alpha, _, _) in enumerate(_weights(_model_key(case))):
        at, k = x.kernel(d, s)
        out[at] = (k @ _dev(alpha)).detach()
    return out
