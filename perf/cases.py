"""Performance cases: the calls a user of this package makes, at the sizes they are made at.

The kinds of work, each through a public entry point:

* ``md``      a molecular-dynamics step on device positions: neighbor list, energy, forces
              and stress of the mapped model (autograd.energy_forces_stress), in the
              mixed-precision form or in FP64; B2 or B3 descriptors.
* ``batch``   mixed-precision predictions of many uneven cells in one call
              (SparseGP.predict_mapped_batched): screening, validation of a training set.
* ``pair``    PairFLARE.compute on LAMMPS's host arrays (ghost atoms, full list with a
              skin), FP64 (its default) or mixed.
* ``mean``    SparseGP.predict_mean, the kernel form of a model that is still being trained.
* ``sor``     SparseGP.predict_SOR, mean and variance of energy, forces and stress: what an
              on-the-fly training loop calls on every frame.
* ``uncert``  SparseGP.predict_energy_uncertainty, the per-atom variances of an MD-size frame.
* ``kuf``     the training set's kernel matrix of a batch of cells (fpp_kuf_batched).
* ``desc``    B2.compute_struc with stored derivatives, the first thing done to a training frame.

Lattices, descriptor settings and model sizes are those of flare_pp_gb300/synth.py and of
the tests (FCC a = 4.05 A, BCC a = 3.0 A, rattled by 0.05-0.1 A).  Sparse sets are the
environments of seeded frames of the same lattice and weights are a regularised fit to
Lennard-Jones site energies, computed here in plain torch FP64; the same plain code, which
uses nothing of the package, gives the exact results.

The mixed form computes in 32 bits, so its results go where such results go: into a
single-precision integrator or model (float32).  FP64 results stay FP64.
"""
import math

import numpy as np
import torch

DEV = "cuda"
F64 = torch.float64

FCC = (4.05, ((0, 0, 0), (0, .5, .5), (.5, 0, .5), (.5, .5, 0)))
BCC = (3.0, ((0, 0, 0), (.5, .5, .5)))


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _case(kind, lattice, reps, ns, N, lmax, rc, sparse, **more):
    c = dict(kind=kind, lattice=lattice, n1=reps[0], n2=reps[1], n3=reps[2], n_species=ns, N=N,
             lmax=lmax, rc=rc, sparse=sparse, power=2, cutoff="quadratic", precision="fp64",
             descriptor="B2", rattle=0.05 if lattice == "fcc" and ns == 1 else 0.08, count=1)
    c.update(more)
    return c


def listed():
    return [
        # the smallest MD cell: 108 atoms of aluminium, where launches and waits are the time
        dict(name="md_fcc108_mixed",
             **_case("md", "fcc", (3, 3, 3), 1, 8, 3, 5.0, 50, precision="mixed")),
        # an ordinary alloy cell
        dict(name="md_bcc2000_mixed",
             **_case("md", "bcc", (10, 10, 10), 2, 10, 4, 5.5, 200, precision="mixed")),
        # the benchmark's production MD frame: 32,768 atoms, 2000 sparse environments per species
        dict(name="md_bcc32k_mixed",
             **_case("md", "bcc", (32, 32, 16), 2, 12, 4, 5.5, 2000, precision="mixed")),
        # the large-scale B3 frame: 1,048,576 atoms of aluminium
        dict(name="md_b3_fcc1m_mixed",
             **_case("md", "fcc", (64, 64, 64), 1, 6, 3, 5.0, 500, precision="mixed",
                     descriptor="B3")),
        # the alloy cell in reference precision (relaxations, elastic constants)
        dict(name="md_bcc2000_fp64",
             **_case("md", "bcc", (10, 10, 10), 2, 10, 4, 5.5, 200)),
        # 256 uneven cells of 32-512 atoms in one call
        dict(name="batch_fcc256_mixed",
             **_case("batch", "fcc", (0, 0, 0), 2, 8, 3, 5.0, 200, precision="mixed",
                     rattle=0.1, count=256)),
        # LAMMPS's rank-size domain through the pair style, in its default precision
        dict(name="pair_bcc4394_fp64",
             **_case("pair", "bcc", (13, 13, 13), 2, 8, 3, 5.5, 200)),
        # the kernel form of an MD-size frame
        dict(name="mean_bcc8k",
             **_case("mean", "bcc", (16, 16, 16), 2, 12, 4, 5.5, 1000)),
        # on-the-fly training: mean and variance of one 256-atom frame
        dict(name="sor_fcc256",
             **_case("sor", "fcc", (4, 4, 4), 2, 8, 3, 5.0, 200, rattle=0.1)),
        # per-atom uncertainties of a 4096-atom frame
        dict(name="uncert_bcc4k",
             **_case("uncert", "bcc", (16, 16, 8), 2, 10, 4, 5.5, 1000)),
        # the training set's kernel matrix: 32 cells with energy, force and stress labels
        dict(name="kuf_fcc32",
             **_case("kuf", "fcc", (0, 0, 0), 2, 8, 3, 5.0, 150, rattle=0.1, count=32)),
        # descriptors and stored derivatives of one training frame
        dict(name="desc_fcc108",
             **_case("desc", "fcc", (3, 3, 3), 1, 8, 3, 5.35, 0, rattle=0.03)),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _reps(rng, lattice, lo, hi):
    """Uneven supercell of about a log-uniform number of atoms in [lo, hi]."""
    per = 4 if lattice == "fcc" else 2
    while True:
        n = _logint(rng, lo, hi) / per
        a = max(2, int(round(n ** (1 / 3) * rng.uniform(0.7, 1.4))))
        b = max(2, int(round(math.sqrt(n / a) * rng.uniform(0.8, 1.25))))
        c = max(2, int(round(n / (a * b))))
        if lo / 2 <= a * b * c * per <= hi:
            return a, b, c


def draw(rng):
    kind = rng.choice(["md", "md", "md", "b3", "fp64", "batch", "pair", "mean", "sor", "uncert",
                       "kuf", "desc"])
    lattice = rng.choice(["fcc", "bcc"])
    ns = rng.choice([1, 2, 2, 2, 3])
    N, lmax = rng.choice([(8, 3), (10, 4), (12, 4), (8, 3), (6, 3), (7, 4), (9, 2)])
    if ns == 3:
        N, lmax = rng.choice([(6, 3), (8, 3)])
    more = dict(cutoff=rng.choice(["quadratic", "quadratic", "quadratic", "cosine"]),
                power=rng.choice([2, 2, 2, 1]))
    rc = {"fcc": 5.0, "bcc": 5.5}[lattice]
    if kind == "b3":
        return _case("md", "fcc", _reps(rng, "fcc", 108, 200000), 1, rng.choice([4, 6]), 3, 5.0,
                     _logint(rng, 50, 500), precision="mixed", descriptor="B3")
    if kind in ("md", "fp64"):
        reps = _reps(rng, lattice, 54, 32000 if kind == "md" else 6000)
        return _case("md", lattice, reps, ns, N, lmax, rc, _logint(rng, 40, 800),
                     precision="mixed" if kind == "md" else "fp64", **more)
    if kind == "batch":
        return _case("batch", "fcc", (0, 0, 0), rng.choice([1, 2]), 8, 3, 5.0,
                     _logint(rng, 50, 300), precision="mixed", rattle=0.1,
                     count=_logint(rng, 4, 256))
    if kind == "pair":
        return _case("pair", lattice, _reps(rng, lattice, 250, 6000), ns, N, lmax, rc,
                     _logint(rng, 40, 300), precision=rng.choice(["fp64", "mixed"]), **more)
    if kind == "mean":
        return _case("mean", lattice, _reps(rng, lattice, 108, 8000), ns, N, lmax, rc,
                     _logint(rng, 50, 1000), **more)
    if kind == "sor":
        return _case("sor", lattice, _reps(rng, lattice, 54, 400), ns, rng.choice([6, 8]), 3, rc,
                     _logint(rng, 50, 300), **more)
    if kind == "uncert":
        return _case("uncert", lattice, _reps(rng, lattice, 108, 8000), ns, N, lmax, rc,
                     _logint(rng, 50, 1000), **more)
    if kind == "kuf":
        return _case("kuf", "fcc", (0, 0, 0), rng.choice([1, 2]), rng.choice([6, 8]), 3, 5.0,
                     _logint(rng, 50, 150), rattle=0.1, count=_logint(rng, 4, 32))
    # cutoffs between two neighbor shells
    return _case("desc", lattice, _reps(rng, lattice, 54, 256), rng.choice([1, 2]),
                 rng.choice([6, 8]), 3, {"fcc": 5.35, "bcc": 5.6}[lattice], 0, rattle=0.03)


# ---------------------------------------------------------------------------
# structures
# ---------------------------------------------------------------------------
def _supercell(lattice, reps, rattle, ns, rng, strain=0.0):
    a, basis = FCC if lattice == "fcc" else BCC
    g = np.stack(np.meshgrid(*[np.arange(n) for n in reps], indexing="ij"), -1).reshape(-1, 3)
    pos = (g[:, None, :] + np.array(basis)[None]).reshape(-1, 3) * a
    cell = np.diag([n * a for n in reps]).astype(np.float64)
    if strain:
        e = rng.uniform(-strain, strain, size=(3, 3))
        f = np.eye(3) + 0.5 * (e + e.T)
        cell, pos = cell @ f, pos @ f
    pos = pos + rng.normal(scale=rattle, size=pos.shape)
    species = rng.permutation(np.arange(len(pos)) % ns)
    return cell, species.astype(np.int32), pos


def _cells(count, ns, rattle, rng):
    """Uneven FCC cells of 32..512 atoms, strained by up to 3 %."""
    shapes = [(4 * a * b * c, (a, b, c)) for a in range(1, 9) for b in range(a, 9)
              for c in range(b, 9)]
    out = []
    for n in np.random.default_rng(404).integers(32, 513, size=count):
        reps = min(shapes, key=lambda s: (abs(s[0] - n), s[1]))[1]
        out.append(_supercell("fcc", reps, rattle, ns, rng, strain=0.03))
    return out


def _frames(case, seed):
    rng = np.random.default_rng([int(seed), 1])
    if case["kind"] in ("batch", "kuf"):
        return _cells(case["count"], case["n_species"], case["rattle"], rng)
    return [_supercell(case["lattice"], (case["n1"], case["n2"], case["n3"]), case["rattle"],
                       case["n_species"], rng)]


def _neighbors(cell, pos, rc):
    """All (i, j, shift) with |x_j - x_i + shift cell| < rc over wrapped positions, in (i, j,
    shift) order, and the vectors: plain FP64, every pair."""
    C = torch.as_tensor(cell, dtype=F64, device=DEV)
    x = torch.as_tensor(pos, dtype=F64, device=DEV)
    frac = x @ torch.linalg.inv(C)
    wrap = torch.floor(frac)
    frac = frac - wrap
    n = len(x)
    vol = float(abs(np.linalg.det(cell)))
    h = [vol / np.linalg.norm(np.cross(cell[(k + 1) % 3], cell[(k + 2) % 3])) for k in range(3)]
    parts = []
    if min(h) > 2 * rc + 0.5:  # the nearest image only
        rows = max(1, min(n, int(3e7) // n))
        for b in range(0, n, rows):
            d = frac[None, :, :] - frac[b:b + rows, None, :]
            s = -torch.round(d)
            v = (d + s) @ C
            m = (v.square().sum(-1) < rc * rc)
            m[torch.arange(m.shape[0]), torch.arange(b, b + m.shape[0])] = False
            i, j = torch.nonzero(m, as_tuple=True)
            parts.append((i + b, j, s[i, j].long(), v[i, j]))
    else:
        reach = [int(math.floor(rc / hk + 1)) for hk in h]
        d = frac[None, :, :] - frac[:, None, :]
        for s1 in range(-reach[0], reach[0] + 1):
            for s2 in range(-reach[1], reach[1] + 1):
                for s3 in range(-reach[2], reach[2] + 1):
                    s = torch.tensor([s1, s2, s3], dtype=F64, device=DEV)
                    v = (d + s) @ C
                    r2 = v.square().sum(-1)
                    i, j = torch.nonzero((r2 < rc * rc) & (r2 > 1e-12), as_tuple=True)
                    parts.append((i, j, s.long().expand(len(i), 3), v[i, j]))
    i, j, s, v = (torch.cat(p) for p in zip(*parts))
    key = (((i * n + j) * 64 + s[:, 0] + 32) * 64 + s[:, 1] + 32) * 64 + s[:, 2] + 32
    o = torch.argsort(key)
    return i[o], j[o], s[o], v[o], wrap


def _padded(i, v, sj, j, n):
    """Pairs (sorted by i) as an n x K table: vectors, neighbor species (-1: none), neighbors."""
    cnt = torch.bincount(i, minlength=n)
    k = torch.arange(len(i), device=DEV) - (torch.cumsum(cnt, 0) - cnt)[i]
    K = max(1, int(cnt.max()) if n else 1)
    V = torch.ones((n, K, 3), dtype=F64, device=DEV)
    S = torch.full((n, K), -1, dtype=torch.long, device=DEV)
    J = torch.zeros((n, K), dtype=torch.long, device=DEV)
    V[i, k], S[i, k], J[i, k] = v, sj, j
    return V, S, J


# ---------------------------------------------------------------------------
# descriptors, plain FP64 torch
# ---------------------------------------------------------------------------
def _harmonics(v, lmax):
    """Orthonormal real harmonics (no Condon-Shortley phase) at l*l + l + m."""
    u = v / v.norm(dim=-1, keepdim=True)
    x, y, z = u[..., 0], u[..., 1], u[..., 2]
    Y = [None] * (lmax + 1) ** 2
    A, B = torch.ones_like(x), torch.zeros_like(x)
    for m in range(lmax + 1):
        if m:
            A, B = x * A - y * B, y * A + x * B
        q1 = q2 = None
        for l in range(m, lmax + 1):
            if l == m:
                q = torch.full_like(x, float(math.prod(range(1, 2 * m, 2))))
            elif l == m + 1:
                q = (2 * m + 1) * z * q1
            else:
                q = ((2 * l - 1) * z * q1 - (l + m - 1) * q2) / (l - m)
            q2, q1 = q1, q
            nrm = math.sqrt((2 * l + 1) / (4 * math.pi) * math.factorial(l - m)
                            / math.factorial(l + m))
            if m == 0:
                Y[l * l + l] = nrm * q
            else:
                Y[l * l + l + m] = math.sqrt(2) * nrm * q * A
                Y[l * l + l - m] = math.sqrt(2) * nrm * q * B
    return torch.stack(Y, -1)


def _radial(r, rc, N, cutoff):
    """Chebyshev x cutoff functions on [0, rc] and their derivatives."""
    x = r / rc
    t, d = [torch.ones_like(r), x], [torch.zeros_like(r), torch.ones_like(r) / rc]
    for n in range(2, N):
        t.append(2 * x * t[-1] - t[-2])
        d.append(2 * t[n - 1] / rc + 2 * x * d[-1] - d[-2])
    t, d = torch.stack(t[:N], -1), torch.stack(d[:N], -1)
    if cutoff == "quadratic":
        f, df = (r - rc).square(), 2 * (r - rc)
    else:
        f = 0.5 * (torch.cos(math.pi * r / rc) + 1)
        df = -0.5 * math.pi / rc * torch.sin(math.pi * r / rc)
    return t * f[..., None], d * f[..., None] + t * df[..., None]


def _bases(case, V, S, grad):
    """Radial rows in their species' block (n, K, ns N), harmonics (n, K, H) and, with grad,
    the radial derivatives, unit vectors and harmonic gradients (n, K, 3, H)."""
    ns, N = case["n_species"], case["N"]
    r = V.norm(dim=-1)
    g, dg = _radial(r, case["rc"], N, case["cutoff"])
    live = ((S >= 0) & (r <= case["rc"]))[..., None]
    block = (S[..., None, None] == torch.arange(ns, device=DEV)[:, None]) & live[..., None]

    def place(q):
        return (q[..., None, :] * block).reshape(*q.shape[:2], ns * N)

    Y = _harmonics(V, case["lmax"])
    if not grad:
        return place(g), Y
    dY = torch.stack([torch.func.jvp(lambda w: _harmonics(w, case["lmax"]), (V,),
                                     (torch.eye(3, dtype=F64, device=DEV)[k].expand_as(V),))[1]
                      for k in range(3)], 2)
    return place(g), Y, place(dg), V / r[..., None], dY


def _single_bond(G, Y):
    return torch.einsum("akn,akh->anh", G, Y)


def _b2(c, lmax):
    i, j = torch.triu_indices(c.shape[1], c.shape[1], device=DEV)
    return torch.stack([torch.einsum("anm,akm->ank", c[:, :, l * l:(l + 1) ** 2],
                                     c[:, :, l * l:(l + 1) ** 2])[:, i, j]
                        for l in range(lmax + 1)], -1).flatten(1)


def _wigner3j(l1, l2, l3, m1, m2, m3):
    f = math.factorial
    if m1 + m2 + m3 or abs(m3) > l3:
        return 0.0
    s = 0.0
    for k in range(max(0, l2 - l3 - m1, l1 - l3 + m2), min(l1 + l2 - l3, l1 - m1, l2 + m2) + 1):
        s += (-1) ** k / (f(k) * f(l3 - l2 + k + m1) * f(l3 - l1 + k - m2) * f(l1 + l2 - l3 - k)
                          * f(l1 - k - m1) * f(l2 - k + m2))
    pre = (f(l1 + l2 - l3) * f(l1 - l2 + l3) * f(-l1 + l2 + l3) / f(l1 + l2 + l3 + 1)
           * f(l1 + m1) * f(l1 - m1) * f(l2 + m2) * f(l2 - m2) * f(l3 + m3) * f(l3 - m3))
    return (-1.0) ** (l1 - l2 - m3) * math.sqrt(pre) * s


def _b3(c, lmax):
    """Re sum_m W c c c over radial triples n1 <= n2 <= n3 and triangles (l1, l2, l3)."""
    z = [None] * c.shape[2]
    for l in range(lmax + 1):
        o = l * l + l
        z[o] = torch.complex(c[..., o], torch.zeros_like(c[..., o]))
        for m in range(1, l + 1):
            R, Sn = c[..., o + m] / math.sqrt(2), c[..., o - m] / math.sqrt(2)
            z[o + m] = (-1) ** m * torch.complex(R, Sn)
            z[o - m] = torch.complex(R, -Sn)
    z = torch.stack(z, -1)
    nr = c.shape[1]
    tri = [(a, b, d) for a in range(nr) for b in range(a, nr) for d in range(b, nr)]
    t1, t2, t3 = (torch.tensor(q, device=DEV) for q in zip(*tri))
    cols = []
    for l1 in range(lmax + 1):
        for l2 in range(lmax + 1):
            for l3 in range(abs(l1 - l2), min(lmax, l1 + l2) + 1):
                W = torch.tensor([[[_wigner3j(l1, l2, l3, a, b, d) for d in range(-l3, l3 + 1)]
                                   for b in range(-l2, l2 + 1)] for a in range(-l1, l1 + 1)],
                                 dtype=torch.complex128, device=DEV)
                T = torch.einsum("mno,axm,ayn->axyo", W, z[..., l1 * l1:(l1 + 1) ** 2],
                                 z[..., l2 * l2:(l2 + 1) ** 2])
                cols.append((T[:, t1, t2] * z[:, t3, l3 * l3:(l3 + 1) ** 2]).sum(-1).real)
    return torch.stack(cols, -1).flatten(1)


def _descriptor(case, c):
    return (_b3 if case["descriptor"] == "B3" else _b2)(c, case["lmax"])


def _environment(case, cell, species, pos):
    """Padded neighbor table of a frame: vectors, neighbor species, neighbors."""
    i, j, _, v, _ = _neighbors(cell, pos, case["rc"])
    sp = torch.as_tensor(species, dtype=torch.long, device=DEV)
    return _padded(i, v, sp[j], j, len(species)) + (sp,)


def _chunks(case, n):
    step = 256 if case["descriptor"] == "B3" else 1024
    return [slice(b, min(n, b + step)) for b in range(0, n, step)]


# ---------------------------------------------------------------------------
# the model: sparse set from seeded frames, weights fitted to Lennard-Jones site energies
# ---------------------------------------------------------------------------
SIGMA, NOISE, SIGMA_E = 2.0, 0.1, 0.5


def _model(case, seed):
    ns, per = case["n_species"], case["sparse"]
    rng = np.random.default_rng([int(seed), 2])
    atoms = 4 if case["lattice"] == "fcc" else 2
    n = max(4, math.ceil((1.15 * per * ns / atoms + 8) ** (1 / 3)))
    cell, species, pos = _supercell(case["lattice"], (n, n, n), case["rattle"], ns, rng)
    V, S, _, sp = _environment(case, cell, species, pos)
    p = torch.cat([_descriptor(case, _single_bond(*_bases(case, V[q], S[q], False)))
                   for q in _chunks(case, len(pos))])
    r = V.norm(dim=-1)
    sr6, cut6 = (2.6 / r) ** 6, (2.6 / case["rc"]) ** 6
    y = (0.8 * ((sr6 * sr6 - sr6) - (cut6 * cut6 - cut6)) * (S >= 0)).sum(1)
    D, nrm, alpha, Ri, Li = [], [], [], [], []
    for s in range(ns):
        idx = torch.nonzero(sp == s).flatten()
        pick = np.sort(rng.permutation(len(idx))[:per])
        d = p[idx[torch.as_tensor(pick, device=DEV)]]
        ys = y[idx[torch.as_tensor(pick, device=DEV)]]
        D.append(d)
        nrm.append(d.norm(dim=1))
        dh = d / nrm[-1][:, None]
        K = SIGMA ** 2 * (dh @ dh.T) ** case["power"]
        eye = torch.eye(len(d), dtype=F64, device=DEV)
        L = torch.linalg.cholesky(K + NOISE ** 2 * eye)
        alpha.append(torch.cholesky_solve(ys[:, None], L)[:, 0])
        if case["kind"] in ("sor", "uncert"):
            Li.append(torch.linalg.solve_triangular(L, eye, upper=False))
            R = torch.linalg.cholesky(K + NOISE ** 2 * eye + K @ K / SIGMA_E ** 2)
            Ri.append(torch.linalg.solve_triangular(R, eye, upper=False).T)
    m = dict(D=D, norms=nrm, alpha=alpha, dhat=[d / n_[:, None] for d, n_ in zip(D, nrm)])
    if Li:
        m.update(R_inv=torch.block_diag(*Ri), L_inv=torch.block_diag(*Li))
    return m


def _descriptor_calculator(case):
    from flare_pp_gb300 import B2, B3
    args = ("chebyshev", case["cutoff"], [0.0, case["rc"]], [],
            [case["n_species"], case["N"], case["lmax"]])
    return (B3 if case["descriptor"] == "B3" else B2)(*args)


def _sparse_gp(case, seed):
    """The trained model as a program has it in hand."""
    from flare_pp_gb300 import ClusterDescriptor, NormalizedDotProduct, SparseGP
    m = _model(case, seed)
    desc = _descriptor_calculator(case)
    cd = ClusterDescriptor()
    cd.initialize_cluster(case["n_species"], desc.n_descriptors)
    cd.descriptors = [d.cpu().numpy() for d in m["D"]]
    cd.descriptor_norms = [d.cpu().numpy() for d in m["norms"]]
    cd.cutoff_values = [np.ones(len(d)) for d in m["D"]]
    cd.n_clusters_by_type = [len(d) for d in m["D"]]
    cd.cumulative_type_count = [int(k) for k in
                                np.cumsum([0] + cd.n_clusters_by_type)[:case["n_species"]]]
    cd.n_clusters = sum(cd.n_clusters_by_type)
    gp = SparseGP([NormalizedDotProduct(SIGMA, case["power"])], 0.01, 0.05, 0.006)
    inv = {k: m[k].cpu().numpy() for k in ("R_inv", "L_inv") if k in m}
    gp.set_model(desc, cd, torch.cat(m["alpha"]).cpu().numpy(), **inv)
    return gp


def _lammps_arrays(case, cell, species, pos):
    """Owned atoms, the ghosts (every periodic image whose lattice site is within the list's
    reach of the box), and a full list with a skin."""
    i, j, s, _, wrap = _neighbors(cell, pos, case["rc"] + 0.3)
    n = len(species)
    s = (s + wrap[i] - wrap[j]).long()  # images of the atoms as they are, not wrapped
    _, _, site = _supercell(case["lattice"], (case["n1"], case["n2"], case["n3"]), 0.0, 1,
                            np.random.default_rng(0))
    box, reach = np.diag(cell), case["rc"] + 1.5
    m = [int(math.ceil(reach / b)) for b in box]
    img = np.stack(np.meshgrid(*[np.arange(-k, k + 1) for k in m], indexing="ij"), -1)
    img = img.reshape(-1, 1, 3)
    at = site[None] + img * box
    near = ((at >= -reach) & (at < box + reach)).all(-1) & (img != 0).any(-1)
    gk, gj = np.nonzero(near)
    index = np.full(near.shape, -1)
    index[gk, gj] = n + np.arange(len(gj))
    index[len(img) // 2] = np.arange(n)
    s, j = s.cpu().numpy(), j.cpu().numpy()
    w = 2 * np.array(m) + 1
    nb = index[((s[:, 0] + m[0]) * w[1] + s[:, 1] + m[1]) * w[2] + s[:, 2] + m[2], j]
    x = np.concatenate([pos, pos[gj] + img[gk, 0] * box])
    return dict(x=x, type_=(species[np.concatenate([np.arange(n), gj])] + 1).astype(np.int32),
                ilist=np.arange(n, dtype=np.int32),
                numneigh=torch.bincount(i, minlength=n).cpu().numpy().astype(np.int32),
                neighbors=nb.astype(np.int32), nlocal=n)


# ---------------------------------------------------------------------------
def prepare(case, seed):
    from flare_pp_gb300 import PairFLARE, Structure, _lib
    kind = case["kind"]
    st = dict(kind=kind, precision=case["precision"], frames=_frames(case, seed))
    cell, species, pos = st["frames"][0]
    if kind == "desc":
        st["b2"] = _descriptor_calculator(case)
        st["structure"] = Structure(cell, species, pos, case["rc"])
        return st
    gp = st["gp"] = _sparse_gp(case, seed)
    if kind == "pair":
        # the mapped coefficients, loaded once as pair_coeff does
        gp.center_mixed_on(Structure(cell, species, pos, case["rc"]))
        st["pair"] = PairFLARE(model=gp._model)
        st["arrays"] = _lammps_arrays(case, cell, species, pos)
        return st
    st["structures"] = [Structure(c, s, p, case["rc"]) for c, s, p in st["frames"]]
    st["structure"] = st["structures"][0]
    if kind in ("md", "batch"):
        # coefficients mapped and centred before the run starts
        gp.center_mixed_on(st["structures"][-1])
        st["positions"] = torch.as_tensor(pos, dtype=F64, device=DEV)
    if kind == "kuf":
        ctypes = _lib.ctypes
        n = [s.noa for s in st["structures"]]
        st["labels"] = sum(1 + 3 * k + 6 for k in n)
        st["handles"] = (ctypes.c_void_p * len(n))(*[s.handle for s in st["structures"]])
        st["mask"] = np.full(len(n), 7, dtype=np.int32)
        st["n_sparse"] = gp.sparse_descriptors[0].n_clusters
    return st


def _single(*arrays):
    """Mixed-precision results as a single-precision consumer keeps them."""
    return [a.float() if isinstance(a, torch.Tensor) else np.asarray(a, dtype=np.float32)
            for a in arrays]


def run(st):
    kind, gp = st["kind"], st.get("gp")
    if kind == "md":
        from flare_pp_gb300.autograd import energy_forces_stress
        out = energy_forces_stress(gp, st["structure"], st["positions"], st["precision"])
        return _single(*out) if st["precision"] == "mixed" else list(out)
    if kind == "batch":
        e, f, s = gp.predict_mapped_batched(st["structures"], "mixed")
        return [e.astype(np.float32), np.concatenate(f, dtype=np.float32), s.astype(np.float32)]
    if kind == "pair":
        f, e, v = st["pair"].compute(precision=st["precision"], **st["arrays"])
        return _single(e, f, v) if st["precision"] == "mixed" else [float(e), f, v]
    if kind == "mean":
        gp.predict_mean(st["structure"])
        return [st["structure"].mean_efs]
    if kind == "sor":
        gp.predict_SOR(st["structure"])
        return [st["structure"].mean_efs, st["structure"].variance_efs]
    if kind == "uncert":
        e, v, local = gp.predict_energy_uncertainty(st["structure"])
        return [float(e), float(v), local]
    if kind == "kuf":
        from flare_pp_gb300._lib import check, lib, ptr
        K = np.empty((st["n_sparse"], st["labels"]))
        check(lib().fpp_kuf_batched(gp._model.handle, st["handles"], len(st["structures"]),
                                    ptr(st["mask"]), None, None, ptr(K), st["labels"], None))
        return [K]
    dv = st["b2"].compute_struc(st["structure"])
    return dict(descriptors=dv.descriptors, norms=dv.descriptor_norms,
                dervs=dv.descriptor_force_dervs, dots=dv.descriptor_force_dots,
                counts=dv.neighbor_counts, coordinates=dv.neighbor_coordinates)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    kind, ns, N = case["kind"], case["n_species"], case["N"]
    if kind in ("batch", "kuf"):
        atoms = 272 * case["count"]
    else:
        atoms = case["n1"] * case["n2"] * case["n3"] * (4 if case["lattice"] == "fcc" else 2)
    per_volume = 4 / 4.05 ** 3 if case["lattice"] == "fcc" else 2 / 27.0
    nb = per_volume * 4 / 3 * math.pi * case["rc"] ** 3
    H, nr, S = (case["lmax"] + 1) ** 2, ns * N, case["sparse"]
    if case["descriptor"] == "B3":
        l = range(case["lmax"] + 1)
        tri = [(a, b, c) for a in l for b in l for c in l if abs(a - b) <= c <= a + b]
        n_d = nr * (nr + 1) * (nr + 2) // 6 * len(tri)
        couple = 8 * (nr * (nr + 1) // 2) * sum((2 * a + 1) * (2 * b + 1) for a, b, _ in tri)
    else:
        n_d = nr * (nr + 1) // 2 * (case["lmax"] + 1)
        couple = nr * (nr + 1) * H
    forward = atoms * (nb * 2 * N * H + couple)
    backward = atoms * (nb * 4 * N * H + 2 * couple)
    if kind == "desc":
        rows = atoms * nb * 3
        return dict(bytes=24 * atoms + 8 * n_d * (atoms + rows),
                    flops=forward + rows * 4 * (nr * (nr + 1) // 2) * H / max(1, ns))
    if kind in ("md", "batch", "pair"):
        size = 4 if case["precision"] == "mixed" else 8
        model = ns * (n_d * n_d if case["power"] == 2 else n_d) * size
        return dict(bytes=model + 48 * atoms,
                    flops=forward + backward + atoms * (2 * n_d * n_d if case["power"] == 2 else 4 * n_d))
    model = 8 * ns * S * n_d
    if kind == "mean":
        return dict(bytes=model + 48 * atoms, flops=forward + backward + atoms * 4 * S * n_d)
    if kind == "uncert":
        return dict(bytes=model + 32 * atoms + 8 * ns * S * S,
                    flops=forward + atoms * (2 * S * n_d + S * S))
    # a kernel matrix: per sparse environment of the atom's species, u = (W + W^T) c and f.dc
    out = ns * S * (1 + 3 * atoms + (6 * case["count"]))
    rows = atoms * S * (4 * n_d + 2 * nr * nr * H + nb * (4 * N * H + 8 * H))
    if kind == "kuf":
        return dict(bytes=model + 24 * atoms + 8 * out, flops=forward + rows)
    n = ns * S
    return dict(bytes=model + 72 * atoms + 8 * n * n, flops=forward + rows + n * n * (1 + 3 * atoms + 6))


# ---------------------------------------------------------------------------
# exact results, plain FP64 torch
# ---------------------------------------------------------------------------
def _site_energies(case, m, p, sp):
    """E_i = sigma^2 sum_k alpha_k (dhat_k . phat_i)^power of a chunk."""
    ph = p / p.norm(dim=1, keepdim=True)
    e = torch.zeros(len(p), dtype=F64, device=DEV)
    for s in range(case["n_species"]):
        z = ph @ m["dhat"][s].T
        e = e + (sp == s) * (SIGMA ** 2 * (z ** case["power"]) @ m["alpha"][s])
    return e


def _pair_forces(u, bases):
    """dE_i/dr_ij = u_i . dc_i/dr_ij for every entry of the padded table (u: a x n x h)."""
    G, Y, dG, rhat, dY = bases
    a = torch.einsum("akn,anh->akh", G, u)
    b = (torch.einsum("akn,anh->akh", dG, u) * Y).sum(-1)
    return torch.einsum("akh,akch->akc", a, dY) + b[..., None] * rhat


def _efs_pairs(case, m, V, S, sp):
    """Site energies and pair forces of a frame."""
    es, fs = [], []
    for q in _chunks(case, len(sp)):
        bases = _bases(case, V[q], S[q], True)
        c = _single_bond(bases[0], bases[1]).requires_grad_(True)
        e = _site_energies(case, m, _descriptor(case, c), sp[q])
        (u,) = torch.autograd.grad(e.sum(), c)
        es.append(e.detach())
        fs.append(_pair_forces(u, bases))
    return torch.cat(es), torch.cat(fs)


def _efs(case, m, cell, species, pos):
    V, S, J, sp = _environment(case, cell, species, pos)
    e, f = _efs_pairs(case, m, V, S, sp)
    F = f.sum(1)
    F = F.index_add(0, J.flatten(), -(f * (S >= 0)[..., None]).reshape(-1, 3))
    W = -torch.einsum("aki,akj->ij", f, V) / abs(np.linalg.det(cell))
    return e.sum(), F, W[[0, 0, 0, 1, 1, 2], [0, 1, 2, 1, 2, 2]]


def _kernel_columns(case, m, cell, species, pos):
    """Kernel of every sparse environment with the frame's energy, forces and stress."""
    V, S, J, sp = _environment(case, cell, species, pos)
    n, lmax = len(species), case["lmax"]
    vol = abs(np.linalg.det(cell))
    nr = case["n_species"] * case["N"]
    i1, i2 = torch.triu_indices(nr, nr, device=DEV)
    bases = _bases(case, V, S, True)
    c = _single_bond(bases[0], bases[1])
    p = _b2(c, lmax)
    nrm = p.norm(dim=1)
    ph = p / nrm[:, None]
    out = []
    for s in range(case["n_species"]):
        at = torch.nonzero(sp == s).flatten()
        mine = [b[at] for b in bases]
        for dh in torch.split(m["dhat"][s], 16):
            z = dh @ ph[at].T
            K = torch.zeros((len(dh), 1 + 3 * n + 6), dtype=F64, device=DEV)
            K[:, 0] = SIGMA ** 2 * (z ** case["power"]).sum(1)
            a = SIGMA ** 2 * case["power"] * z ** (case["power"] - 1) / nrm[at]
            w = a[..., None] * (dh[:, None] - z[..., None] * ph[at])
            w = w.reshape(len(dh), len(at), -1, lmax + 1)
            W = torch.zeros((len(dh), len(at), nr, nr, lmax + 1), dtype=F64, device=DEV)
            W[:, :, i1, i2] += w
            W[:, :, i2, i1] += w
            u = torch.cat([torch.einsum("xanm,amh->xanh", W[..., l],
                                        c[at][:, :, l * l:(l + 1) ** 2])
                           for l in range(lmax + 1)], -1)
            for k in range(len(dh)):
                f = _pair_forces(u[k], mine)
                F = torch.zeros((n, 3), dtype=F64, device=DEV)
                F[at] = f.sum(1)
                F = F.index_add(0, J[at].flatten(),
                                -(f * (S[at] >= 0)[..., None]).reshape(-1, 3))
                Wt = -torch.einsum("aki,akj->ij", f, V[at]) / vol
                K[k, 1:1 + 3 * n] = F.flatten()
                K[k, 1 + 3 * n:] = Wt[[0, 0, 0, 1, 1, 2], [0, 1, 2, 1, 2, 2]]
            out.append(K)
    return torch.cat(out)


def _exact_desc(case, cell, species, pos):
    i, j, _, v, _ = _neighbors(cell, pos, case["rc"])
    sp = torch.as_tensor(species, dtype=torch.long, device=DEV)
    V, S, _ = _padded(i, v, sp[j], j, len(species))
    lmax, nr = case["lmax"], case["n_species"] * case["N"]
    bases = _bases(case, V, S, True)
    G, Y, dG, rhat, dY = bases
    c = _single_bond(G, Y)
    p = _b2(c, lmax)
    live = S >= 0
    dc = (torch.einsum("akn,akc,akh->akcnh", dG, rhat, Y)
          + torch.einsum("akn,akch->akcnh", G, dY))[live]
    ca = c[torch.nonzero(live)[:, 0]]
    i1, i2 = torch.triu_indices(nr, nr, device=DEV)
    dp = []
    for l in range(lmax + 1):
        q = slice(l * l, (l + 1) ** 2)
        t = torch.einsum("pcnm,pkm->pcnk", dc[..., q], ca[..., q])
        dp.append((t + t.transpose(-1, -2))[..., i1, i2])
    dp = torch.stack(dp, -1).flatten(2)
    dots = (dp * p[i][:, None, :]).sum(-1)
    cnt = torch.bincount(i, minlength=len(species))
    out = dict(descriptors=[], norms=[], dervs=[], dots=[], counts=[], coordinates=[])
    for s in range(case["n_species"]):
        at, rows = sp == s, sp[i] == s
        out["descriptors"].append(p[at])
        out["norms"].append(p[at].norm(dim=1))
        out["dervs"].append(dp[rows].flatten(0, 1))
        out["dots"].append(dots[rows].flatten())
        out["counts"].append(cnt[at])
        out["coordinates"].append(v[rows])
    return out


def exact(case, seed):
    kind = case["kind"]
    frames = _frames(case, seed)
    if sum(len(s) for _, s, _ in frames) > 300000:
        return None  # a million B3 environments take minutes in plain FP64
    cell, species, pos = frames[0]
    if kind == "desc":
        return _exact_desc(case, cell, species, pos)
    m = _model(case, seed)
    if kind == "md":
        return list(_efs(case, m, cell, species, pos))
    if kind == "batch":
        got = [_efs(case, m, *fr) for fr in frames]
        return [torch.stack([g[0] for g in got]), torch.cat([g[1] for g in got]),
                torch.stack([g[2] for g in got])]
    if kind == "pair":
        a = _lammps_arrays(case, cell, species, pos)
        n = a["nlocal"]
        x = torch.as_tensor(a["x"], device=DEV)
        j = torch.as_tensor(a["neighbors"], dtype=torch.long, device=DEV)
        i = torch.repeat_interleave(torch.arange(n, device=DEV),
                                    torch.as_tensor(a["numneigh"], dtype=torch.long, device=DEV))
        v = x[j] - x[i]
        keep = v.square().sum(1) < case["rc"] ** 2
        i, j, v = i[keep], j[keep], v[keep]
        kinds = torch.as_tensor(a["type_"], dtype=torch.long, device=DEV) - 1
        V, S, J = _padded(i, v, kinds[j], j, n)
        e, f = _efs_pairs(case, m, V, S, kinds[:n])
        f = f * (S >= 0)[..., None]
        F = torch.zeros((len(x), 3), dtype=F64, device=DEV)
        F[:n] = f.sum(1)
        F = F.index_add(0, J.flatten(), -f.reshape(-1, 3))
        W = -torch.einsum("aki,akj->ij", V, f)
        return [e.sum(), F, W[[0, 1, 2, 0, 0, 1], [0, 1, 2, 1, 2, 2]]]
    if kind == "mean":
        e, F, W = _efs(case, m, cell, species, pos)
        return [torch.cat([e[None], F.flatten(), W])]
    if kind == "sor":
        K = _kernel_columns(case, m, cell, species, pos)
        return [K.T @ torch.cat(m["alpha"]), (m["R_inv"].T @ K).square().sum(0)]
    if kind == "kuf":
        return [torch.cat([_kernel_columns(case, m, *fr) for fr in frames], 1)]
    V, S, _, sp = _environment(case, cell, species, pos)
    p = torch.cat([_descriptor(case, _single_bond(*_bases(case, V[q], S[q], False)))
                   for q in _chunks(case, len(pos))])
    ph = p / p.norm(dim=1, keepdim=True)
    k = torch.cat([(SIGMA ** 2 * (ph @ d.T) ** case["power"]) * (sp == s)[:, None]
                   for s, d in enumerate(m["dhat"])], 1)
    kE = k.sum(0)
    local = SIGMA ** 2 - (k @ m["L_inv"].T).square().sum(1)
    return [kE @ torch.cat(m["alpha"]), (m["R_inv"].T @ kE).square().sum(), local]
