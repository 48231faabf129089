"""The calls that a user of this framework makes, for timing and comparison.

Sizes and distributions are those of the repository's own workloads
(gapgb/synth.py, bench.py, tests/): the 64-atom Si and C cells, the 512-atom
ternary alloy, the ragged structure-search population, the Si/Ge MD cell, the
variance and fit of the alloy model, the surrogate of the alloy descriptors.
`exact` states the same quantities in 64 bits with plain torch: wACSF
descriptors, the sparse GPR, forces and stress through autograd, the normal
equations of the fit, and the committee networks.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "calypso-gap_gb300"))

RCUT = 6.0
PI = 3.141592654          # the cutoff function's pi (a model constant of the format)
GPA = 6.24219e-3          # eV / A^3 per GPa, likewise
KB, ACCEL, KINETIC = 8.617333262e-5, 9.648533212331e-3, 103.642697
MASS = {14: 28.0855, 32: 72.630}
DEV = "cuda"
F64 = torch.float64


# ---------------------------------------------------------------- the cases

def listed():
    return [
        # one call of the drop-in calculator on a small cell in the default
        # FP64 form, as an ASE relaxation makes it at every step
        dict(name="cell_si64", kind="cell", proto="si", reps="2x2x2", sf="std", M=500, grad=True),
        # the same with the reference example's symmetry functions: seven
        # angular cutoffs, 158 neighbours per atom, a small model
        dict(name="cell_carbon64", kind="cell", proto="c", reps="2x2x2", sf="multi", M=129,
             grad=True),
        # the same on the 512-atom alloy cell with a full-size model
        dict(name="cell_alloy512", kind="cell", proto="alloy", reps="4x4x8", sf="std", M=4000,
             grad=True),
        # a set of uneven candidate cells in the FP64 form: final energies,
        # forces and atomic energies of a search's survivors
        dict(name="batch_ragged_fp64", kind="batch", cells=48, nmin=8, nmax=256, M=2000,
             precision="fp64"),
        # the headline screening step: equal cells, tensor-core form, device buffers
        dict(name="screen_alloy_tc", kind="device", cells=76, reps="4x4x8", M=4000,
             precision="tc"),
        # a structure-search generation from host buffers, 8 to 256 atoms a cell
        dict(name="search_population_tc", kind="batch", cells=1024, nmin=8, nmax=256, M=4000,
             precision="tc"),
        # ten steps of NVE dynamics of the large Si/Ge cell, one list rebuild among them
        dict(name="md_sige_tc", kind="md", reps=16, M=8000, steps=10, precision="tc"),
        # predictive variance of a batch, for choosing what to label next
        dict(name="variance_alloy_tc", kind="variance", cells=32, M=4000, precision="tc"),
        # refitting the coefficients: energies of many cells
        dict(name="fit_energies_alloy", kind="fit", proto="alloy", reps="4x4x8", cells=48, M=1500,
             forces=False),
        # and energies, forces and stresses of a few small ones
        dict(name="fit_forces_si", kind="fit", proto="si", reps="2x2x2", cells=8, M=150,
             forces=True),
        # one training step of the surrogate committee (forward, backward, Adam)
        dict(name="surrogate_train", kind="train", cells=16, rows=1024, hidden=128, members=4),
        # the committee's prediction for a batch
        dict(name="surrogate_predict", kind="predict", cells=64, hidden=128, members=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cell", "cell", "cell", "batch", "batch", "device", "md", "variance", "fit",
                       "fit", "train", "predict"])
    if kind == "cell":
        proto = rng.choice(["si", "c", "alloy"])
        top = {"si": 3, "c": 2, "alloy": 6}[proto]
        reps = "x".join(str(rng.randint(1, top)) for _ in range(3))
        return dict(kind=kind, proto=proto, reps=reps, sf="multi" if proto == "c" else "std",
                    M=_log(rng, 129, 4000) if proto != "c" else _log(rng, 65, 500),
                    grad=rng.random() < 0.85)
    if kind == "batch":
        prec = rng.choice(["fp64", "fp64", "mixed", "fp32", "tc", "tf32"])
        top = 64 if prec in ("fp64", "mixed") else 768
        nmax = rng.randint(40, 256)
        return dict(kind=kind, cells=_log(rng, 2, top), nmin=rng.randint(3, 32), nmax=nmax,
                    M=_log(rng, 200, 2400), precision=prec)
    if kind == "device":
        return dict(kind=kind, cells=_log(rng, 1, 76), reps="4x4x%d" % rng.choice([4, 6, 8]),
                    M=_log(rng, 500, 4000), precision=rng.choice(["tc", "tc", "tf32", "fp32"]))
    if kind == "md":
        return dict(kind=kind, reps=rng.randint(3, 14), M=_log(rng, 500, 8000),
                    steps=rng.randint(4, 12), precision=rng.choice(["tc", "tc", "fp32"]))
    if kind == "variance":
        return dict(kind=kind, cells=_log(rng, 1, 32), M=_log(rng, 300, 3000),
                    precision=rng.choice(["tc", "tc", "fp32"]))
    if kind == "fit":
        if rng.random() < 0.5:
            return dict(kind=kind, proto="si", reps="2x2x%d" % rng.randint(1, 3),
                        cells=rng.randint(2, 8), M=_log(rng, 30, 120), forces=True)
        return dict(kind=kind, proto="alloy", reps="4x4x%d" % rng.randint(4, 8),
                    cells=_log(rng, 6, 48), M=_log(rng, 200, 1500), forces=False)
    if kind == "train":
        return dict(kind=kind, cells=rng.randint(4, 16), rows=64 * rng.randint(2, 16), hidden=128,
                    members=rng.choice([2, 4]))
    return dict(kind=kind, cells=_log(rng, 1, 64), hidden=128, members=rng.choice([2, 4]))


# ------------------------------------------------------------ symmetry functions

def sf_table(which):
    """(type, alpha, cutoff, zeta) rows.  std: 20 radial and 12 angular
    functions with one cutoff; multi: the reference example's 33 rows."""
    rows = []
    if which == "std":
        rows += [(1, float(a), 6.0, 1.0) for a in np.geomspace(0.003, 2.0, 20)]
        rows += [(t, a, 6.0, z) for z in (1.0, 2.0, 4.0) for t in (2, 4) for a in (0.003, 0.03)]
    else:
        cuts = (6.0, 2.0, 1.5, 5.0, 4.0, 3.5, 3.0)
        rows += [(1, a, 6.0, 1.0) for a in (1.0, 0.5, 0.1, 0.05, 0.01, 0.005, 0.001)]
        rows += [(2, 0.01, c, 1.0) for c in cuts]
        rows += [(3, a, 6.0, 1.0) for a in (3.0, 2.5, 2.0, 1.5, 1.0)]
        rows += [(2, 0.1, c, 1.0) for c in cuts]
        rows += [(4, 0.01, c, 1.0) for c in cuts]
    t, a, c, z = zip(*rows)
    return (np.array(t, np.int32), np.array(a), np.array(c), np.array(z))


def weights_of(species):
    """Species table: atomic-number weights, carbon as the reference example has it."""
    z = np.array(sorted(species), np.int32)
    return z, np.where(z == 6, 4.0, z.astype(np.float64))


# ------------------------------------------------------------------- structures

def _reps(text):
    return tuple(int(v) for v in text.split("x"))


FCC = np.array([[0, 0, 0], [0, .5, .5], [.5, 0, .5], [.5, .5, 0]])
PROTO = {"si": (np.concatenate([FCC, FCC + .25]), 5.43, 0.05, (14,), (1.0,)),
         "c": (np.concatenate([FCC, FCC + .25]), 3.556, 0.1, (6,), (1.0,)),
         "alloy": (FCC, 3.9, 0.08, (13, 28, 40), (0.5, 0.3, 0.2)),
         "sige": (np.concatenate([FCC, FCC + .25]), 5.54, 0.1, (14, 32), (0.5, 0.5))}


def crystal(proto, reps, rng):
    """(lat, pos, z): a jittered, randomly occupied crystal."""
    basis, a, jitter, elems, frac = PROTO[proto]
    g = np.stack(np.meshgrid(*[np.arange(n) for n in reps], indexing="ij"), -1).reshape(-1, 1, 3)
    lat = np.diag([a * n for n in reps]).astype(np.float64)
    pos = ((g + basis[None]).reshape(-1, 3) * a) + rng.normal(0.0, jitter, (g.shape[0] * len(basis), 3))
    n = len(pos)
    counts = [int(round(f * n)) for f in frac[:-1]]
    z = np.repeat(np.array(elems, np.int32), counts + [n - sum(counts)])
    rng.shuffle(z)
    return lat, pos, z


def pack(structs):
    off = np.cumsum([0] + [len(p) for _, p, _ in structs]).astype(np.int32)
    return (off, np.concatenate([z for _, _, z in structs]).astype(np.int32),
            np.stack([l for l, _, _ in structs]), np.concatenate([p for _, p, _ in structs]))


def random_cells(count, nmin, nmax, seed):
    """Random triclinic cells (angles 60-120 degrees, 12-20 A^3 per atom, no
    two atoms within 1.6 A, 1-4 species of {3, 8, 14, 26}): every cell is
    filled at once, one accepted atom a round."""
    rng = np.random.default_rng(seed)
    pool = np.array([3, 8, 14, 26], np.int32)
    shifts = np.stack(np.meshgrid([-1, 0, 1], [-1, 0, 1], [-1, 0, 1], indexing="ij"), -1).reshape(-1, 3)
    ns = np.random.default_rng(count).integers(nmin, nmax + 1, count).tolist()  # of the case
    lats, elems = [], []
    for n in ns:
        while True:
            ca, cb, cg = np.cos(np.radians(rng.uniform(60, 120, 3)))
            if 1 - ca * ca - cb * cb - cg * cg + 2 * ca * cb * cg <= 0.05:
                continue
            a, b, c = rng.uniform(0.8, 1.25, 3)
            sg = math.sqrt(1 - cg * cg)
            cx, cy = c * cb, c * (ca - cb * cg) / sg
            lat = np.array([[a, 0, 0], [b * cg, b * sg, 0],
                            [cx, cy, math.sqrt(max(c * c - cx * cx - cy * cy, 1e-12))]])
            lat = lat * (n * rng.uniform(12, 20) / abs(np.linalg.det(lat))) ** (1 / 3)
            if np.sqrt(((shifts[np.abs(shifts).sum(1) > 0] @ lat) ** 2).sum(1)).min() >= 1.6:
                break
        lats.append(lat)
        elems.append(rng.choice(pool, int(rng.integers(1, 5)), replace=False))
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(rng.integers(1 << 40)))
    want = torch.tensor(ns, device=DEV)
    L = torch.tensor(np.stack(lats), dtype=torch.float32, device=DEV)
    sh = torch.tensor(shifts, dtype=torch.float32, device=DEV)
    frac = torch.full((count, nmax, 3), 0.5, dtype=torch.float32, device=DEV)
    have = torch.zeros(count, dtype=torch.long, device=DEV)
    rows = torch.arange(count, device=DEV)
    slot = torch.arange(nmax, device=DEV)
    while bool((have < want).any()):
        f = torch.rand((count, 3), generator=gen, device=DEV)
        d = frac - f[:, None, :]
        d = d - d.round()
        near = torch.full((count, nmax), 1e9, device=DEV)
        for s in sh:
            near = torch.minimum(near, torch.einsum("cna,cab->cnb", d + s, L).square().sum(-1))
        near = torch.where(slot[None] < have[:, None], near, torch.full_like(near, 1e9))
        ok = (near.amin(1) >= 1.6002 ** 2) & (have < want)
        frac[rows[ok], have[ok]] = f[ok]
        have = have + ok.long()
    frac = frac.double().cpu().numpy()
    out = []
    for k in range(count):
        z = elems[k][rng.integers(0, len(elems[k]), ns[k])].astype(np.int32)
        out.append((lats[k], frac[k, :ns[k]] @ lats[k], z))
    return out


# --------------------------------------------------- the same quantities in 64 bits

def neighbours(lat, pos):
    """Every (i, j, p_j + n L - r_i) within RCUT, sorted by i."""
    lat = torch.as_tensor(lat, dtype=F64, device=DEV)
    pos = torch.as_tensor(pos, dtype=F64, device=DEV)
    inv = torch.linalg.inv(lat)
    width = RCUT * inv.square().sum(0).sqrt()
    n = pos.shape[0]
    frac = pos @ inv
    chunk = max(1, 4_000_000 // n)
    got = []
    if float(width.max()) < 0.5:      # the nearest image is the only one within reach
        for a in range(0, n, chunk):
            d = frac[None] - frac[a:a + chunk, None]
            v = pos[None] - pos[a:a + chunk, None] - d.round() @ lat
            hit = v.square().sum(-1) <= RCUT * RCUT
            hit[torch.arange(hit.shape[0]), torch.arange(a, a + hit.shape[0])] = False
            i, j = torch.nonzero(hit, as_tuple=True)
            got.append((i + a, j, v[i, j]))
    else:
        top = [int(math.ceil(float(w) + 1.0)) for w in width]
        grid = [torch.arange(-t, t + 1, dtype=F64, device=DEV) for t in top]
        sh = torch.cartesian_prod(*grid) @ lat
        home = pos - frac.floor() @ lat      # images are counted from the home cell
        for s in range(0, sh.shape[0], max(1, 8_000_000 // (n * n))):
            t = sh[s:s + max(1, 8_000_000 // (n * n))]
            v = home[None, None] + t[:, None, None] - home[None, :, None]
            r2 = v.square().sum(-1)
            k, i, j = torch.nonzero((r2 <= RCUT * RCUT) & (r2 > 1e-16), as_tuple=True)
            got.append((i, j, v[k, i, j]))
    i, j, v = (torch.cat(x) for x in zip(*got))
    order = torch.argsort(i, stable=True)
    return i[order], j[order], v[order]


def padded(lists, n):
    """(vec[n, P, 3], j[n, P], real[n, P]) of sorted neighbour triples; unused
    slots lie far from everything."""
    i, j, v = lists
    count = torch.bincount(i, minlength=n)
    P = max(2, int(count.max()))
    q = torch.arange(i.shape[0], device=DEV) - (count.cumsum(0) - count)[i]
    vec = torch.zeros((n, P, 3), dtype=F64, device=DEV)
    vec[..., 0] = 100.0 + 20.0 * torch.arange(P, device=DEV, dtype=F64)
    vec[i, q] = v
    jj = torch.zeros((n, P), dtype=torch.long, device=DEV)
    jj[i, q] = j
    real = torch.zeros((n, P), dtype=torch.bool, device=DEV)
    real[i, q] = True
    return vec, jj, real


def wacsf(vec, w, sf):
    """Descriptors [n, 2 nsf] of padded slots (differentiable in vec)."""
    ty, al, rc, ze = sf
    n, P, _ = vec.shape
    zero = torch.zeros((), dtype=F64, device=DEV)

    def cut(r, c):
        return torch.where(r <= c, 0.5 * (torch.cos(PI / c * r) + 1.0), zero)

    r = vec.square().sum(-1).sqrt()
    nsf = len(ty)
    G = [None] * (2 * nsf)
    jj, kk = torch.triu_indices(P, P, 1, device=DEV)
    a, b = r[:, jj], r[:, kk]
    c = (vec[:, jj] - vec[:, kk]).square().sum(-1).sqrt()
    cos = (a * a + b * b - c * c) / (2.0 * a * b)
    s3 = a * a + b * b + c * c
    ww = w[:, jj] * w[:, kk]
    fc = {}
    ex = {}
    for s in range(nsf):
        t, x, cu, zeta = int(ty[s]), float(al[s]), float(rc[s]), float(ze[s])
        if t in (1, 3):
            v = (torch.exp(-x * r * r) if t == 1 else torch.exp(-4.0 * (r - x) ** 2)) * cut(r, cu)
            G[s], G[s + nsf] = v.sum(1), (v * w).sum(1)
            continue
        if cu not in fc:
            one = cut(r, cu)
            fc[cu] = one[:, jj] * one[:, kk] * cut(c, cu)
        if x not in ex:
            ex[x] = torch.exp(-x * s3)
        base = 1.0 + cos if t == 2 else 1.0 - cos
        v = 2.0 ** (1.0 - zeta) * base ** int(zeta) * ex[x] * fc[cu]
        G[s], G[s + nsf] = v.sum(1), (v * ww).sum(1)
    return torch.stack(G, 1)


def gpr(G, theta, mm, coeff):
    """Atomic energies and dE/dG of the sparse GPR, by direct differences."""
    th, m, c = (torch.as_tensor(v, dtype=F64, device=DEV) for v in (theta, mm, coeff))
    mu = m.mean(0)
    mt = ((m - mu) / th).contiguous()
    e = torch.empty(G.shape[0], dtype=F64, device=DEV)
    dg = torch.empty_like(G)
    step = max(1, 16_000_000 // m.shape[0])
    for a in range(0, G.shape[0], step):
        x = (G[a:a + step] - mu) / th
        wk = torch.exp(-0.5 * dist2(x, mt)) * c
        e[a:a + step] = wk.sum(1)
        dg[a:a + step] = -(x * wk.sum(1, keepdim=True) - wk @ mt) / th
    return e, dg


def dist2(x, m):
    s = torch.zeros((x.shape[0], m.shape[0]), dtype=F64, device=DEV)
    for d in range(x.shape[1]):
        s += (x[:, d, None] - m[None, :, d]).square()
    return s


def lists_of(batch):
    off, sp, lat, pos = batch
    got = []
    for s in range(len(off) - 1):
        i, j, v = neighbours(lat[s], pos[off[s]:off[s + 1]])
        got.append((i + int(off[s]), j + int(off[s]), v))
    return tuple(torch.cat(x) for x in zip(*got))


def atom_weights(sp, table):
    w = dict(zip(table[0].tolist(), table[1].tolist()))
    return torch.tensor([w[int(z)] for z in sp], dtype=F64, device=DEV)


def chunks_of(lists, n):
    """Ranges of atoms whose padded triples stay within memory."""
    count = torch.bincount(lists[0], minlength=n)
    start = torch.cat([torch.zeros(1, dtype=torch.long, device=DEV), count.cumsum(0)]).cpu().numpy()
    P = max(2, int(count.max()))
    step = max(1, 4_000_000 // (P * (P - 1) // 2))
    for a in range(0, n, step):
        b = min(n, a + step)
        yield a, b, int(start[a]), int(start[b])


def descriptors(batch, sf, table, lists=None):
    n = int(batch[0][-1])
    lists = lists_of(batch) if lists is None else lists
    w = atom_weights(batch[1], table)
    out = []
    for a, b, s, t in chunks_of(lists, n):
        vec, jj, _ = padded((lists[0][s:t] - a, lists[1][s:t], lists[2][s:t]), b - a)
        out.append(wacsf(vec, w[jj], sf))
    return torch.cat(out)


def pull(batch, sf, table, lists, dedg):
    """(forces [N, 3], stress [S, 6] GPa) of the descriptor gradient dedg."""
    off, sp, lat, pos = batch
    n, S = int(off[-1]), len(off) - 1
    w = atom_weights(sp, table)
    cell = torch.repeat_interleave(torch.arange(S, device=DEV),
                                   torch.as_tensor(np.diff(off), device=DEV))
    F = torch.zeros((n, 3), dtype=F64, device=DEV)
    vir = torch.zeros((S, 3, 3), dtype=F64, device=DEV)
    for a, b, s, t in chunks_of(lists, n):
        vec, jj, real = padded((lists[0][s:t] - a, lists[1][s:t], lists[2][s:t]), b - a)
        vec.requires_grad_(True)
        G = wacsf(vec, w[jj], sf)
        g, = torch.autograd.grad((G * dedg[a:b]).sum(), vec)
        g = torch.where(real[..., None], g, torch.zeros_like(g))
        v = torch.where(real[..., None], vec.detach(), torch.zeros_like(g))
        F[a:b] += g.sum(1)
        F.index_add_(0, jj[real], -g[real])
        vir.index_add_(0, cell[a:b], torch.einsum("npa,npb->nab", v, g))
    vol = torch.as_tensor(np.abs(np.linalg.det(lat)), device=DEV)
    st = -vir / vol[:, None, None] / GPA
    return F, torch.stack([st[:, 0, 0], st[:, 1, 1], st[:, 2, 2], st[:, 0, 1], st[:, 1, 2],
                           st[:, 0, 2]], 1)


def evaluate(batch, arrays, grad=True):
    """(E [S], F [N, 3], stress [S, 6], e [N])."""
    table, sf, theta, mm, coeff = arrays
    lists = lists_of(batch)
    e, dg = gpr(descriptors(batch, sf, table, lists), theta, mm, coeff)
    S = len(batch[0]) - 1
    cell = torch.repeat_interleave(torch.arange(S, device=DEV),
                                   torch.as_tensor(np.diff(batch[0]), device=DEV))
    E = torch.zeros(S, dtype=F64, device=DEV).index_add_(0, cell, e)
    if not grad:
        return E, torch.zeros((e.shape[0], 3), dtype=F64), torch.zeros((S, 6), dtype=F64), e
    F, st = pull(batch, sf, table, lists, dg)
    return E, F, st, e


# ----------------------------------------------------------------------- models

def gpr_arrays(batch, sf, table, M, scale, seed):
    """theta, mm, coeff: M sparse points drawn from the batch's descriptors,
    length scales that follow their spread."""
    rng = np.random.default_rng(seed)
    X = descriptors(batch, sf, table).cpu().numpy()
    mm = X[rng.choice(len(X), size=M, replace=len(X) < M)].copy()
    sd = mm.std(0)
    return np.where(sd > 1e-9, scale * sd, 1.0), mm, rng.normal(0.0, 1e-3, M)


@functools.lru_cache(maxsize=None)
def model_arrays(proto, sfname, M):
    """(species table, SF table, theta, mm, coeff): the model a program loads."""
    rng = np.random.default_rng(97)
    if proto == "population":
        cells, species = random_cells(max(4, -(-M // 100)), 8, 256, 97), (3, 8, 14, 26)
    else:
        reps = {"si": (2, 2, 2), "c": (2, 2, 2), "alloy": (4, 4, 8), "sige": (8, 8, 8)}[proto]
        count = max(1, -(-M // (len(PROTO[proto][0]) * reps[0] * reps[1] * reps[2])))
        cells, species = [crystal(proto, reps, rng) for _ in range(count)], PROTO[proto][3]
    sf, table = sf_table(sfname), weights_of(species)
    theta, mm, coeff = gpr_arrays(pack(cells), sf, table, M, 0.8 if proto == "alloy" else 1.0, 5)
    return table, sf, theta, mm, coeff


def handle(arrays, precision, cap=None):
    import gapgb
    (z, w), (ty, al, rc, ze), theta, mm, coeff = arrays
    m = gapgb.GapModel.create(z, w, ty, al, rc, theta, mm, coeff, sf_zeta=ze, rcut=RCUT)
    m.set_precision(precision)
    if cap:
        m.set_neighbour_cap(cap)
    return m


@functools.lru_cache(maxsize=2)
def qmm_of(M):
    """(K_MM + 0.01 I)^-1 of the alloy model."""
    _, _, theta, mm, _ = model_arrays("alloy", "std", M)
    x = torch.as_tensor((mm - mm.mean(0)) / theta, device=DEV)
    K = torch.exp(-0.5 * dist2(x, x)) + 0.01 * torch.eye(M, dtype=F64, device=DEV)
    return torch.cholesky_inverse(torch.linalg.cholesky(K)).cpu().numpy()


# ------------------------------------------------------------------------ inputs

def the_batch(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "cell":
        return pack([crystal(case["proto"], _reps(case["reps"]), rng)])
    if kind == "batch":
        return pack(random_cells(case["cells"], case["nmin"], case["nmax"], seed))
    if kind == "device":
        return pack([crystal("alloy", _reps(case["reps"]), rng) for _ in range(case["cells"])])
    if kind == "fit":
        return pack([crystal(case["proto"], _reps(case["reps"]), rng) for _ in range(case["cells"])])
    if kind == "md":
        return pack([crystal("sige", (case["reps"],) * 3, rng)])
    return pack([crystal("alloy", (4, 4, 8), rng) for _ in range(case["cells"])])


def arrays_of(case):
    kind = case["kind"]
    if kind == "cell":
        return model_arrays(case["proto"], case["sf"], case["M"])
    return model_arrays({"batch": "population", "md": "sige"}.get(kind, "alloy"), "std", case["M"])


def velocities(z, seed):
    """Maxwell-Boltzmann at 600 K, no net momentum."""
    rng = np.random.default_rng(seed + 1)
    m = np.array([MASS[int(v)] for v in z])
    v = rng.normal(0.0, 1.0, (len(m), 3)) * np.sqrt(KB * 600.0 / (m * KINETIC))[:, None]
    return m, v - (m[:, None] * v).sum(0) / m.sum()


# noise levels that leave the coefficients determined by the data to about ten
# digits (at 1 meV per atom the alloy set's normal matrix leaves seven)
SIGMA = dict(sigma_e=2e-2, sigma_f=0.1, sigma_s=0.1, jitter=1e-6)


def fit_data(case, seed):
    """Training set and its labels: a smooth pair energy of the cells, its
    forces and stress; the sparse points are taken from the set itself."""
    batch = the_batch(case, seed)
    off, sp, lat, pos = batch
    table, sf = weights_of(PROTO[case["proto"]][3]), sf_table("std")
    some = -(-case["M"] // int(off[1]))
    head = int(off[min(some, len(off) - 1)])
    part = (off[:min(some, len(off) - 1) + 1], sp[:head], lat[:min(some, len(off) - 1)], pos[:head])
    theta, mm, _ = gpr_arrays(part, sf, table, case["M"],
                              0.8 if case["proto"] == "alloy" else 1.0, seed)
    S, n = len(off) - 1, int(off[-1])
    v, _, real = padded(lists_of(batch), n)      # sums in a fixed order: the labels repeat
    r = v.square().sum(-1).sqrt()
    w = torch.where(real, (1 - (r / RCUT).square()), torch.zeros_like(r))
    bell = -0.4 * torch.exp(-(r - 2.5).square())
    de = bell * w * (-2.0 * (r - 2.5) * w - 4.0 * r / RCUT ** 2)
    E = (0.5 * bell * w * w).sum(1).reshape(S, -1).sum(1)
    f = (de / r)[..., None] * v
    F = f.sum(1)
    vir = (0.5 * v[..., :, None] * f[..., None, :]).sum(1).reshape(S, -1, 3, 3).sum(1)
    st = -vir / torch.as_tensor(np.abs(np.linalg.det(lat)), device=DEV)[:, None, None] / GPA
    st = torch.stack([st[:, 0, 0], st[:, 1, 1], st[:, 2, 2], st[:, 0, 1], st[:, 1, 2], st[:, 0, 2]], 1)
    return batch, table, sf, theta, mm, E.cpu().numpy(), F.cpu().numpy(), st.cpu().numpy()


def layout(D, H):
    """Offsets of one network's parameters and the block size."""
    sizes = [("W1", (H, D)), ("b1", (H,)), ("W2", (H, H)), ("b2", (H,)), ("w3", (H,)), ("b3", (1,))]
    at, out = 0, {}
    for name, shape in sizes:
        out[name] = (at, shape)
        at += int(np.prod(shape))
    return out, -(-at // 8) * 8


def surrogate_data(case, seed):
    """Labels of alloy atoms (descriptors, energies, dE/dG of a smooth GAP),
    their standardisation, and weights as a fresh committee has them."""
    batch = the_batch(case, seed)
    table, sf, theta, mm, coeff = model_arrays("alloy", "std", 1000)
    G = descriptors(batch, sf, table)
    e, t = gpr(G, 5.0 * theta, mm, coeff)
    G32, t32 = G.float(), t.float()
    Z = torch.as_tensor(batch[1], device=DEV)
    rng = np.random.default_rng(seed + 2)
    zs = table[0].tolist()
    shift = [float(e[Z == z].mean()) for z in zs]
    scale = float(torch.cat([e[Z == z] - s for z, s in zip(zs, shift)]).std())
    norm = (G32.double().mean(0).cpu().numpy(), G32.double().std(0).cpu().numpy(),
            np.array(shift), scale)
    H, Q = case["hidden"], case["members"]
    lay, P = layout(G.shape[1], H)
    W = np.zeros((Q, len(zs), P), np.float32)
    for name, (at, shape) in lay.items():
        size = int(np.prod(shape))
        if name in ("W1", "W2", "w3"):
            W[:, :, at:at + size] = rng.normal(0.0, 1.0 / math.sqrt(shape[-1]), (Q, len(zs), size))
    rows = None
    if case["kind"] == "train":
        rows = np.stack([np.stack([rng.choice(np.flatnonzero(batch[1] == z), case["rows"],
                                              replace=True) for z in zs]) for _ in range(Q)])
        rows = torch.as_tensor(rows.astype(np.int32), device=DEV)
    return zs, Z, G32.contiguous(), e, t32.contiguous(), norm, W, rows


LAM, LR = 1.0, 2e-3


def prepare(case, seed):
    kind = case["kind"]
    if kind == "cell":
        off, sp, lat, pos = the_batch(case, seed)
        return dict(case=case, model=handle(arrays_of(case), "fp64"), sp=sp, lat=lat[0], pos=pos)
    if kind == "batch":
        return dict(case=case, model=handle(arrays_of(case), case["precision"]),
                    batch=the_batch(case, seed))
    if kind == "device":
        off, sp, lat, pos = the_batch(case, seed)
        S, n = len(off) - 1, int(off[-1])
        return dict(case=case, model=handle(arrays_of(case), case["precision"], 96), S=S, n=n,
                    most=int(np.diff(off).max()),
                    dev=[torch.as_tensor(v, device=DEV).contiguous() for v in (off, sp, lat, pos)],
                    out=[torch.empty(s, dtype=F64, device=DEV) for s in ((S,), (n, 3), (S, 6))])
    if kind == "md":
        from gapgb.md import MD
        off, sp, lat, pos = the_batch(case, seed)
        mass, vel = velocities(sp, seed)
        model = handle(arrays_of(case), case["precision"], 64)
        return dict(case=case, model=model, md=MD(model, off, sp, lat, pos, vel, mass, dt=1.0,
                                                  skin=0.5, rebuild_every=10))
    if kind == "variance":
        m = handle(arrays_of(case), case["precision"])
        m.set_qmm(qmm_of(case["M"]))
        return dict(case=case, model=m, batch=the_batch(case, seed))
    if kind == "fit":
        batch, table, sf, theta, mm, E, F, st = fit_data(case, seed)
        m = handle((table, sf, theta, mm, np.zeros(case["M"])), "fp64")
        return dict(case=case, model=m, batch=batch, E=E, F=F, st=st)
    from gapgb.surrogate import Surrogate
    zs, Z, G, e, t, norm, W, rows = surrogate_data(case, seed)
    sur = Surrogate(zs, G.shape[1], hidden=case["hidden"], members=case["members"], seed=0)
    sur.set_norm(*norm)
    sur.set_params(W)
    n = G.shape[0]
    out = [torch.empty(n, dtype=F64, device=DEV), torch.empty(n, dtype=torch.float32, device=DEV),
           torch.empty_like(G)]
    return dict(case=case, sur=sur, Z=Z, G=G, e=e, t=t, rows=rows, out=out,
                grad=torch.empty(W.shape, dtype=torch.float32, device=DEV))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "cell":
        E, F, st, var = state["model"].eval(state["sp"], state["lat"], state["pos"], case["grad"])
        return dict(E=E, F=F, stress=st)
    if kind == "batch":
        E, F, st, e = state["model"].eval_batch(*state["batch"], lgrad=True, atom_energy=True)
        return dict(E=E, F=F, stress=st, e=e)
    if kind == "device":
        off, sp, lat, pos = state["dev"]
        E, F, st = state["out"]
        state["model"].eval_batch_ptrs(state["S"], state["n"], state["most"], off.data_ptr(),
                                       sp.data_ptr(), lat.data_ptr(), pos.data_ptr(), True,
                                       E.data_ptr(), F.data_ptr(), st.data_ptr(),
                                       stream=torch.cuda.current_stream().cuda_stream)
        return dict(E=E, F=F, stress=st)
    if kind == "md":
        md = state["md"]
        ep, ek = md.run(case["steps"])
        return dict(epot=ep, ekin=ek, pos=md.t["pos"], vel=md.t["vel"])
    if kind == "variance":
        covf, var = state["model"].variance(*state["batch"])
        return dict(covf=covf, var=var)
    if kind == "fit":
        if case["forces"]:
            return state["model"].fit(*state["batch"], state["E"], forces=state["F"],
                                      stress=state["st"], **SIGMA)
        return state["model"].fit_energies(*state["batch"], state["E"], sigma_e=SIGMA["sigma_e"],
                                           jitter=SIGMA["jitter"])
    sur = state["sur"]
    if kind == "train":
        sur.train_step_ptrs(case["rows"], state["rows"].data_ptr(), state["G"].data_ptr(),
                            state["e"].data_ptr(), state["t"].data_ptr(), LAM, LR, True, False,
                            state["grad"].data_ptr())
        return state["grad"]
    e, sd, dg = state["out"]
    sur.predict_ptrs(state["G"].shape[0], state["Z"].data_ptr(), state["G"].data_ptr(),
                     e.data_ptr(), sd.data_ptr(), dg.data_ptr(),
                     torch.cuda.current_stream().cuda_stream)
    return dict(e=e, std=sd, dedg=dg)


# -------------------------------------------------------------------------- work

def atoms_of(case):
    kind = case["kind"]
    if kind == "batch":
        return case["cells"] * (case["nmin"] + case["nmax"]) // 2
    if kind == "md":
        return 8 * case["reps"] ** 3
    if kind in ("variance", "train", "predict"):
        return case["cells"] * 512
    per = len(PROTO[case.get("proto", "alloy")][0])
    return case.get("cells", 1) * per * int(np.prod(_reps(case["reps"])))


def work(case):
    """Counted once: positions, species and lattices in, results out, the
    model's arrays; the GPR contraction (4 M D an atom), the angular pairs
    within the cutoff (about 60 operations for a value, 120 for a gradient)
    and the radial terms."""
    kind, n = case["kind"], atoms_of(case)
    D, M = 64 if case.get("sf") != "multi" else 66, case.get("M", 0)
    slots, pairs = {"c": (158, 5600), "si": (46, 480), "sige": (44, 440)}.get(case.get("proto") or (
        "sige" if kind == "md" else ""), (56, 690))
    io = n * (28 + 24 + 8) + M * D * 8
    desc = n * (pairs * 60 + slots * 200)
    full = desc + n * (pairs * 120 + slots * 200) + 4.0 * n * M * D
    if kind == "cell":
        return dict(bytes=io, flops=full if case["grad"] else desc + 2.0 * n * M * D)
    if kind in ("batch", "device"):
        return dict(bytes=io, flops=full)
    if kind == "md":
        return dict(bytes=case["steps"] * (n * 48 + io), flops=case["steps"] * full)
    if kind == "variance":
        return dict(bytes=io + M * M * 8, flops=desc + 2.0 * n * M * M + 2.0 * n * M * D)
    if kind == "fit":
        S = case["cells"]
        rows = S + (3 * n + 6 * S if case["forces"] else 0)
        fl = desc + 2.0 * n * M * D + rows * float(M) * M + M ** 3 / 3.0
        if case["forces"]:
            fl += M * n * pairs * 120.0
        return dict(bytes=io + rows * 8, flops=fl)
    H, Q = case["hidden"], case["members"]
    net = 2.0 * (D * H + H * H)
    if kind == "train":
        r = 3 * case["rows"]
        P = layout(64, H)[1]
        return dict(bytes=Q * (r * (D * 8 + 8) + 3 * P * 4 * 5), flops=Q * r * net * 7)
    return dict(bytes=n * (D * 4 + 4 + 12 + D * 4), flops=Q * n * net * 2)


# ------------------------------------------------------------------------- exact

def exact(case, seed):
    kind = case["kind"]
    if kind in ("cell", "batch", "device"):
        E, F, st, e = evaluate(the_batch(case, seed), arrays_of(case), case.get("grad", True))
        if kind == "cell":
            return dict(E=float(E[0]), F=F, stress=st[0])
        out = dict(E=E, F=F, stress=st)
        return dict(out, e=e) if kind == "batch" else out
    if kind == "md":
        return exact_md(case, seed)
    if kind == "variance":
        batch = the_batch(case, seed)
        table, sf, theta, mm, _ = arrays_of(case)
        Q = torch.as_tensor(qmm_of(case["M"]), device=DEV)
        mu = torch.as_tensor(mm.mean(0), device=DEV)
        x = (descriptors(batch, sf, table) - mu) / torch.as_tensor(theta, device=DEV)
        m = (torch.as_tensor(mm, device=DEV) - mu) / torch.as_tensor(theta, device=DEV)
        covf = []
        for a in range(0, x.shape[0], 4096):
            K = torch.exp(-0.5 * dist2(x[a:a + 4096], m))
            covf.append(1.0 - ((K @ Q.T) * K).sum(1))
        covf = torch.cat(covf)
        return dict(covf=covf, var=covf.reshape(case["cells"], -1).mean(1))
    if kind == "fit":
        return exact_fit(case, seed)
    return exact_surrogate(case, seed)


def exact_md(case, seed):
    off, sp, lat, pos = the_batch(case, seed)
    arrays = arrays_of(case)
    mass, vel = velocities(sp, seed)
    L = torch.as_tensor(lat[0], device=DEV)
    inv = torch.linalg.inv(L)
    x, v, m = (torch.as_tensor(t, device=DEV) for t in (pos, vel, mass))

    def wrap(x):
        f = x @ inv
        out = (f.floor() != 0).any(1, keepdim=True)
        return torch.where(out, (f - f.floor()) @ L, x)

    def force(x):
        E, F, _, _ = evaluate((off, sp, lat, x), arrays)
        return E, F

    x = wrap(x)
    E, F = force(x)
    acc = (ACCEL / m)[:, None]
    ep, ek = [], []
    for k in range(1, case["steps"] + 1):
        v = v + 0.5 * acc * F
        x = x + v
        if k % 10 == 0:
            x = wrap(x)
        E, F = force(x)
        v = v + 0.5 * acc * F
        ep.append(E)
        ek.append(0.5 * KINETIC * (m[:, None] * v * v).sum().reshape(1))
    return dict(epot=torch.stack(ep), ekin=torch.stack(ek), pos=x, vel=v)


def exact_fit(case, seed):
    batch, table, sf, theta, mm, E, F, st = fit_data(case, seed)
    off = batch[0]
    S, M = len(off) - 1, case["M"]
    lists = lists_of(batch)
    G = descriptors(batch, sf, table, lists)
    th, m = torch.as_tensor(theta, device=DEV), torch.as_tensor(mm, device=DEV)
    mu = m.mean(0)
    x, mt = (G - mu) / th, (m - mu) / th
    cell = torch.repeat_interleave(torch.arange(S, device=DEV), torch.as_tensor(np.diff(off), device=DEV))
    K = torch.exp(-0.5 * dist2(x, mt))
    phi = torch.zeros((S, M), dtype=F64, device=DEV).index_add_(0, cell, K)
    w = torch.as_tensor(1.0 / (SIGMA["sigma_e"] ** 2 * np.diff(off)), device=DEV)
    A = torch.exp(-0.5 * dist2(mt, mt)) + SIGMA["jitter"] * torch.eye(M, dtype=F64, device=DEV)
    A = A + phi.T @ (w[:, None] * phi)
    b = phi.T @ (w * torch.as_tensor(E, device=DEV))
    if case["forces"]:
        PF = torch.empty((3 * x.shape[0], M), dtype=F64, device=DEV)
        PS = torch.empty((6 * S, M), dtype=F64, device=DEV)
        for k in range(M):
            f, s = pull(batch, sf, table, lists, -K[:, k:k + 1] * (x - mt[k]) / th)
            PF[:, k], PS[:, k] = f.reshape(-1), s.reshape(-1)
        A = A + PF.T @ PF / SIGMA["sigma_f"] ** 2 + PS.T @ PS / SIGMA["sigma_s"] ** 2
        b = b + PF.T @ torch.as_tensor(F.reshape(-1), device=DEV) / SIGMA["sigma_f"] ** 2
        b = b + PS.T @ torch.as_tensor(st.reshape(-1), device=DEV) / SIGMA["sigma_s"] ** 2
    return torch.cholesky_solve(b[:, None], torch.linalg.cholesky(A))[:, 0]


def network(p, x, lay):
    """y of one member's network for standardised inputs x."""
    g = {k: p[at:at + int(np.prod(s))].reshape(s) for k, (at, s) in lay.items()}
    a = torch.nn.functional.silu(x @ g["W1"].T + g["b1"])
    return torch.nn.functional.silu(a @ g["W2"].T + g["b2"]) @ g["w3"] + g["b3"]


def exact_surrogate(case, seed):
    zs, Z, G, e, t, (mean, std, shift, scale), W, rows = surrogate_data(case, seed)
    mean, std = torch.as_tensor(mean, device=DEV), torch.as_tensor(std, device=DEV)
    W = torch.as_tensor(W, device=DEV).double()
    lay, P = layout(G.shape[1], case["hidden"])
    Q = case["members"]
    if case["kind"] == "train":
        out = torch.zeros_like(W)
        for q in range(Q):
            for s in range(len(zs)):
                r = rows[q, s].long()
                x = ((G[r].double() - mean) / std).requires_grad_(True)
                p = W[q, s].clone().requires_grad_(True)
                y = network(p, x, lay)
                g, = torch.autograd.grad(y.sum(), x, create_graph=True)
                dy = y - (e[r] - shift[s]) / scale
                dg = g - t[r].double() * std / scale
                loss = (dy.square() + LAM * dg.square().sum(1)).mean()
                out[q, s], = torch.autograd.grad(loss, p)
        return out
    n = G.shape[0]
    y = torch.zeros((Q, n), dtype=F64, device=DEV)
    dg = torch.zeros(G.shape, dtype=F64, device=DEV)
    for s, z in enumerate(zs):
        r = torch.nonzero(Z == z)[:, 0]
        for q in range(Q):
            x = ((G[r].double() - mean) / std).requires_grad_(True)
            v = network(W[q, s], x, lay)
            g, = torch.autograd.grad(v.sum(), x)
            y[q, r] = v.detach() * scale + shift[s]
            dg[r] += g * scale / std / Q
    return dict(e=y.mean(0), std=y.std(0), dedg=dg)
