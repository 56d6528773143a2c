"""Performance cases of the molecular Hartree-Fock path: what programs ask this library for, over the range
in which they ask for it.

  eri       batches of Cartesian ERIs of every (s,p,d) quartet class, device buffers, FP64 or FP32
            (integral consumers, the metric's microbenchmark);
  eri_host  the same through host arrays (a caller without device memory of its own);
  jk        one direct J/K build of a water cluster (an SCF iteration of the caller's own SCF), in an
            uncontracted even-tempered or a contracted split-valence basis, FP64, mixed FP32/FP64, FP32 or
            deterministic;
  rhf       RHF time-to-solution of one new geometry, handle set-up included (a geometry scan);
  rhf_batch the energies of many conformers in one batch handle (a conformer scan);
  mlp       one training step of the learned-guess network.

A case is a dict of plain values; `draw` gives further cases of the same ranges.
"""
import math

import numpy as np
import torch

from qchem_b200 import api, basis

PAIRS = [(0, 0), (1, 0), (1, 1), (2, 0), (2, 1), (2, 2)]
CLASSES = [PAIRS[x] + PAIRS[y] for x in range(6) for y in range(x + 1)]
POOL = 2048                      # random shells per angular momentum of the integral batches
JK_EXACT_NBF = 64                # largest basis whose J and K are rebuilt from a dense ERI tensor


def listed():
    return [
        # integrals of a few quartets of each class on demand: launches and latency
        {"name": "eri_tiny", "kind": "eri", "nq": 32, "precision": "f64"},
        # an ordinary batch, a ragged count
        {"name": "eri_20k", "kind": "eri", "nq": 20011, "precision": "f64"},
        # the microbenchmark's throughput regime
        {"name": "eri_250k", "kind": "eri", "nq": 250000, "precision": "f64"},
        # single-precision integrals
        {"name": "eri_f32_20k", "kind": "eri", "nq": 20011, "precision": "f32"},
        # integrals into host arrays
        {"name": "eri_host_3k", "kind": "eri_host", "nq": 3001, "precision": "f64"},
        # the smallest build: one water, 57 functions
        {"name": "jk_1w", "kind": "jk", "waters": 1, "basis": "even", "mode": "f64"},
        # a mixed-precision build of an ordinary cluster, 228 functions
        {"name": "jk_4w_mixed", "kind": "jk", "waters": 4, "basis": "even", "mode": "mixed"},
        # a contracted split-valence basis, 8 waters, 296 functions
        {"name": "jk_8w_contracted", "kind": "jk", "waters": 8, "basis": "split", "mode": "f64"},
        # a large build: 16 waters, 912 functions
        {"name": "jk_16w", "kind": "jk", "waters": 16, "basis": "even", "mode": "f64"},
        # one RHF of a new geometry, its energy and density
        {"name": "rhf_1w", "kind": "rhf", "waters": 1, "basis": "even"},
        # many conformers at once
        {"name": "rhf_batch_48", "kind": "rhf_batch", "conformers": 48, "basis": "even"},
        # one training step of the learned guess: 128 conformers x 6 atom pairs
        {"name": "mlp_step", "kind": "mlp", "rows": 768, "width": 256},
    ]


def draw(rng):
    kind = rng.choice(["eri", "eri", "eri", "eri_host", "jk", "jk", "jk", "rhf", "rhf_batch", "mlp"])

    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if kind == "eri":
        precision = rng.choice(["f64", "f64", "f32"])
        return {"kind": kind, "nq": spread(1, 250000 if precision == "f64" else 60000), "precision": precision}
    if kind == "eri_host":
        return {"kind": kind, "nq": spread(1, 6000), "precision": rng.choice(["f64", "f32"])}
    if kind == "jk":
        mode = rng.choice(["f64", "f64", "mixed", "f32", "det"])
        largest = {"f64": 14, "mixed": 8, "f32": 1, "det": 8}[mode]
        # a jittered spacing, so that two draws of the same size still differ
        return {"kind": kind, "waters": spread(1, largest), "basis": rng.choice(["even", "split"]), "mode": mode,
                "spacing": round(rng.uniform(5.2, 6.5), 3)}
    if kind == "rhf":
        return {"kind": kind, "waters": 1, "basis": rng.choice(["even", "split"]), "jitter": round(rng.uniform(0.05, 0.15), 3)}
    if kind == "rhf_batch":
        return {"kind": kind, "conformers": spread(2, 64), "basis": rng.choice(["even", "split"]),
                "jitter": round(rng.uniform(0.05, 0.15), 3)}
    return {"kind": "mlp", "rows": spread(6, 1536), "width": rng.choice([128, 192, 256])}


# ------------------------------------------------------------------------------------------------------
# inputs: geometries and shells as plain values (L, centre, exponents, coefficients)
# ------------------------------------------------------------------------------------------------------
WATER = np.array([[0.0, 0.0, 0.0], [1.43, 1.11, 0.0], [-1.43, 1.11, 0.0]])
# even-tempered exponents 0.1 * 2.5^k, k = 0 .. n-1, per element and L
EVEN = {8: {0: 8, 1: 5, 2: 2}, 1: {0: 5, 1: 2}}
# the same exponents contracted to a split-valence set: the k of each shell
SPLIT = {8: {0: [(7, 6, 5), (4, 3, 2), (1,), (0,)], 1: [(4, 3, 2), (1,), (0,)], 2: [(1, 0)]},
         1: {0: [(4, 3, 2), (1,), (0,)], 1: [(1,), (0,)]}}
CONTRACTION = {1: (1.0,), 2: (0.45, 0.65), 3: (0.2, 0.5, 0.45)}


def cluster(case, rng):
    """`waters` waters on a jittered cubic grid, randomly turned: (charges, positions)."""
    n, spacing = case["waters"], case.get("spacing", 5.5)
    side = math.ceil(n ** (1.0 / 3.0) - 1e-9)
    cells = [(i, j, k) for k in range(side) for j in range(side) for i in range(side)][:n]
    Z, R = [], []
    for c in cells:
        w = WATER + rng.uniform(-1.0, 1.0, size=(3, 3)) * case.get("jitter", 0.1)
        q = rng.normal(size=4)
        a, x, y, z = q / np.linalg.norm(q)
        rot = np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - z * a), 2 * (x * z + y * a)],
                        [2 * (x * y + z * a), 1 - 2 * (x * x + z * z), 2 * (y * z - x * a)],
                        [2 * (x * z - y * a), 2 * (y * z + x * a), 1 - 2 * (x * x + y * y)]])
        R.append(np.array(c, float) * spacing + rng.uniform(-0.3, 0.3, size=3) + w @ rot.T)
        Z += [8, 1, 1]
    return Z, np.concatenate(R)


def molecule_shells(kind, Z, R):
    out = []
    for z, r in zip(Z, R):
        for L in sorted(EVEN[z]):
            groups = [(k,) for k in range(EVEN[z][L])] if kind == "even" else SPLIT[z][L]
            out += [(L, tuple(float(v) for v in r), [0.1 * 2.5 ** k for k in g], list(CONTRACTION[len(g)])) for g in groups]
    return out


def pool_shells(rng):
    """random shells: contraction 1-3, exponents log-uniform in [0.05, 50], centres in a 12-bohr box"""
    out = []
    for L in range(3):
        for _ in range(POOL):
            k = int(rng.integers(1, 4))
            out.append((L, tuple(float(v) for v in rng.uniform(0.0, 12.0, size=3)),
                        [float(v) for v in np.exp(rng.uniform(math.log(0.05), math.log(50.0), size=k))],
                        [float(v) for v in rng.uniform(0.1, 1.0, size=k)]))
    return out


def pool_quartets(nq, rng):
    """per class, nq x 4 shell indices into pool_shells"""
    return [np.stack([L * POOL + rng.integers(0, POOL, size=nq) for L in c], axis=1).astype(np.int32) for c in CLASSES]


def density(n, nocc, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    q, _ = torch.linalg.qr(torch.randn(n, nocc, dtype=torch.float64, device="cuda", generator=g))
    return (2.0 * q @ q.T).contiguous()


def nbf_of(shells):
    return sum((s[0] + 1) * (s[0] + 2) // 2 for s in shells)


def block_size(c):
    return math.prod((l + 1) * (l + 2) // 2 for l in c)


def molecules(case, seed):
    """the geometries of an SCF case"""
    rng = np.random.default_rng(seed)
    if case["kind"] == "rhf":
        return [cluster(case, rng)]
    one = dict(case, waters=1)
    return [cluster(one, rng) for _ in range(case["conformers"])]


def mlp_widths(case):
    return [29, case["width"], case["width"], case["width"], 35 * 35]


def mlp_inputs(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    w = mlp_widths(case)
    x = torch.randn(case["rows"], w[0], device="cuda", generator=g)
    t = torch.randn(case["rows"], w[-1], device="cuda", generator=g)
    # the three block shapes of a water's atom pairs, padded to the oxygen's 35 functions
    shapes = [(35, 35), (35, 11), (35, 11), (11, 11), (11, 11), (11, 11)]
    m = torch.zeros(case["rows"], 35, 35, device="cuda")
    for k, (a, b) in enumerate(shapes):
        m[k::6, :a, :b] = 1.0
    p = [v for a, b in zip(w[:-1], w[1:])
         for v in (torch.randn(b, a, device="cuda", generator=g) / math.sqrt(a), 0.01 * torch.randn(b, device="cuda", generator=g))]
    return x, (t * m.reshape(case["rows"], -1)).contiguous(), m.reshape(case["rows"], -1).contiguous(), p


# ------------------------------------------------------------------------------------------------------
# prepare / run
# ------------------------------------------------------------------------------------------------------
def engine(shells):
    e = api.Engine([basis.Shell(*s) for s in shells])
    e.set_stream(torch.cuda.current_stream().cuda_stream)
    return e


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind in ("eri", "eri_host"):
        eng = engine(pool_shells(rng))
        quartets = pool_quartets(case["nq"], rng)
        if kind == "eri_host":
            return {"case": case, "engine": eng, "quartets": quartets}
        t = torch.float64 if case["precision"] == "f64" else torch.float32
        return {"case": case, "engine": eng, "quartets": [torch.from_numpy(q).cuda() for q in quartets],
                "out": [torch.empty(case["nq"], block_size(c), dtype=t, device="cuda") for c in CLASSES]}
    if kind == "jk":
        Z, R = cluster(case, rng)
        eng = engine(molecule_shells(case["basis"], Z, R))
        eng.schwarz(1e-10)
        if case["mode"] == "mixed":
            eng.set_fp32_bound(1e-7)
        D = density(eng.nbf, 5 * case["waters"], seed)
        return {"case": case, "engine": eng, "D": D, "J": torch.empty_like(D), "K": torch.empty_like(D)}
    if kind in ("rhf", "rhf_batch"):
        mols = molecules(case, seed)
        return {"case": case, "mols": [basis.Molecule(Z, R) for Z, R in mols],
                "shells": [[basis.Shell(*s) for s in molecule_shells(case["basis"], Z, R)] for Z, R in mols]}
    x, t, m, p = mlp_inputs(case, seed)
    net = api.Mlp(mlp_widths(case))
    net.set_params(torch.cat([v.reshape(-1) for v in p]).cpu().numpy())
    net.set_stream(torch.cuda.current_stream().cuda_stream)
    return {"case": case, "net": net, "x": x, "t": t, "m": m}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "eri":
        f32 = case["precision"] == "f32"
        for c, q, o in zip(CLASSES, state["quartets"], state["out"]):
            state["engine"].eri_batch_device(c, q.data_ptr(), case["nq"], o.data_ptr(), fp32=f32)
        return state["out"]
    if kind == "eri_host":
        f32 = case["precision"] == "f32"
        return [state["engine"].eri_batch(c, q, fp32=f32) for c, q in zip(CLASSES, state["quartets"])]
    if kind == "jk":
        state["engine"].fock_jk_device(state["D"].data_ptr(), state["J"].data_ptr(), state["K"].data_ptr(),
                                       fp32=case["mode"] == "f32", deterministic=case["mode"] == "det")
        return state["J"], state["K"]
    # DIIS from the first iteration; the scan's energies stop on the density error
    if kind == "rhf":
        r = api.Engine(state["shells"][0]).rhf(state["mols"][0], diis_fdmax=1e6, want_density=True)
        return r["energy"], r["D"]
    if kind == "rhf_batch":
        r = api.BatchEngine(state["shells"]).rhf(state["mols"], fd_tol=1e-7, diis_fdmax=1e6)
        return np.array([x["energy"] for x in r])
    loss, grad = state["net"].loss_grad(case["rows"], state["x"].data_ptr(), state["t"].data_ptr(), state["m"].data_ptr(),
                                        want_grad=True)
    state["net"].adam(lr=1e-3)
    return loss, grad


# ------------------------------------------------------------------------------------------------------
# work
# ------------------------------------------------------------------------------------------------------
def comps(L):
    return [(L - m - l, l, m) for m in range(L + 1) for l in range(L - m + 1)]


def nherm(L):
    return (L + 1) * (L + 2) * (L + 3) // 6


def class_flops(c, prim, bra_prim):
    """Floating-point operations of one contracted quartet with `prim` primitive quartets and `bra_prim` bra
    primitive pairs: Boys and Hermite integrals and the ket contraction to [.|f0) per primitive quartet, the
    bra contraction to [e0|f0] per bra primitive pair, the transfer to (ab|cd) once."""
    la, lb, lc, ld = c
    L, E, F = sum(c), [e for l in range(la, la + lb + 1) for e in comps(l)], [f for l in range(lc, lc + ld + 1) for f in comps(l)]
    support = lambda v: sum((x + 1) * (y + 1) * (z + 1) for x, y, z in v)  # noqa: E731
    ncd = block_size((lc, ld))
    per_prim = 20 + 3 * L + 2 * sum(nherm(j) for j in range(L + 1)) + 2 * nherm(la + lb) * support(F)
    transfer = (2 * len(E) * ncd if ld else 0) + (2 * ncd * block_size((la, lb)) if lb else 0)
    return prim * per_prim + bra_prim * 2 * len(F) * support(E) + transfer


def jk_flops(kind, Z, R):
    """One J/K build: the quartets that survive screening, counted with the Gaussian-product prefactor of a
    pair in place of its Schwarz bound, their integrals and the digestion of each (12 operations)."""
    shells = molecule_shells(kind, Z, R)
    L = np.array([s[0] for s in shells])
    amin = np.array([min(s[2]) for s in shells])
    npr = np.array([len(s[2]) for s in shells])
    cen = np.array([s[1] for s in shells])
    a, b = np.tril_indices(len(shells))
    a, b = np.where(L[a] >= L[b], a, b), np.where(L[a] >= L[b], b, a)
    r2 = ((cen[a] - cen[b]) ** 2).sum(axis=1)
    q = np.exp(-amin[a] * amin[b] / (amin[a] + amin[b]) * r2)
    total = 0.0
    for X in range(6):
        for Y in range(X + 1):
            x, y = (np.flatnonzero((L[a] == p[0]) & (L[b] == p[1])) for p in (PAIRS[X], PAIRS[Y]))
            qy = np.sort(q[y])
            kept = len(qy) - np.searchsorted(qy, 1e-10 / np.maximum(q[x], 1e-300))
            quartets = float(kept.sum()) * (0.5 if X == Y else 1.0)
            if not quartets:
                continue
            bra = float((npr[a] * npr[b])[x].mean())
            ket = float((npr[a] * npr[b])[y].mean())
            c = PAIRS[X] + PAIRS[Y]
            total += quartets * (class_flops(c, bra * ket, bra) + 12 * block_size(c))
    return total


def work(case):
    kind = case["kind"]
    if kind in ("eri", "eri_host"):
        size = 8 if case["precision"] == "f64" else 4
        n = case["nq"]
        # contraction 1-3 per shell: 4 primitive pairs on average
        return {"bytes": float(n * sum(16 + size * block_size(c) for c in CLASSES)),
                "flops": float(n * sum(class_flops(c, 16, 4) for c in CLASSES))}
    if kind == "jk":
        Z, R = cluster(case, np.random.default_rng(0))
        n = nbf_of(molecule_shells(case["basis"], Z, R))
        return {"bytes": 24.0 * n * n, "flops": jk_flops(case["basis"], Z, R)}
    if kind in ("rhf", "rhf_batch"):
        mols = molecules(case, 0)
        n = nbf_of(molecule_shells(case["basis"], *mols[0]))
        # about 15 iterations, each a build and an eigensolve of order n
        one = jk_flops(case["basis"], *mols[0]) + 20.0 * n ** 3
        return {"bytes": 8.0 * n * n * len(mols), "flops": 15.0 * one * len(mols)}
    w = mlp_widths(case)
    params = sum(a * b + b for a, b in zip(w[:-1], w[1:]))
    return {"bytes": 4.0 * (case["rows"] * (w[0] + 2 * w[-1]) + 8 * params), "flops": 6.0 * case["rows"] * params}


# ------------------------------------------------------------------------------------------------------
# exact: the same quantities in plain 64-bit torch and numpy (McMurchie-Davidson, Boys function by series)
# ------------------------------------------------------------------------------------------------------
def boys(n, T):
    """[F_0(T) .. F_n(T)]: the ascending series of F_n and the downward recursion below T = 20, erf and the
    upward recursion above."""
    low = T < 20.0
    t = torch.where(low, T, torch.zeros_like(T))
    term = torch.full_like(t, 1.0 / (2 * n + 1))
    top = term.clone()
    for i in range(1, 110):
        term = term * (2.0 * t / (2 * n + 2 * i + 1))
        top += term
    e = torch.exp(-t)
    down = [None] * n + [top * e]
    for m in range(n - 1, -1, -1):
        down[m] = (2.0 * t * down[m + 1] + e) / (2 * m + 1)
    u = torch.where(low, torch.full_like(T, 20.0), T)
    up, e = [0.5 * torch.sqrt(math.pi / u) * torch.erf(torch.sqrt(u))], torch.exp(-u)
    for m in range(n):
        up.append(((2 * m + 1) * up[m] - e) / (2.0 * u))
    return [torch.where(low, x, y) for x, y in zip(down, up)]


def hermite(la, lb, PA, PB, p):
    """E[i][j][t] of one direction, i <= la, j <= lb, t <= i + j"""
    h = 0.5 / p
    E = [[None] * (lb + 1) for _ in range(la + 1)]
    E[0][0] = [torch.ones_like(p)]

    def raised(src, X):
        n = len(src)
        return [(src[t - 1] * h if t else 0.0) + (src[t] * X if t < n else 0.0) + (src[t + 1] * (t + 1) if t + 1 < n else 0.0)
                for t in range(n + 1)]

    for i in range(la + 1):
        if i:
            E[i][0] = raised(E[i - 1][0], PA)
        for j in range(1, lb + 1):
            E[i][j] = raised(E[i][j - 1], PB)
    return E


def triples(L):
    return [(t, u, v) for t in range(L + 1) for u in range(L + 1 - t) for v in range(L + 1 - t - u)]


def hermite_coulomb(L, alpha, X, Y, Z):
    """R_tuv, t + u + v <= L, stacked in the order of triples(L)"""
    F = boys(L, alpha * (X * X + Y * Y + Z * Z))
    R = {(n, 0, 0, 0): (-2.0 * alpha) ** n * F[n] for n in range(L + 1)}
    for s in range(1, L + 1):
        for t, u, v in triples(s):
            if t + u + v != s:
                continue
            axis, D = (0, X) if t else (1, Y) if u else (2, Z)
            k = (t, u, v)[axis]
            low = [t, u, v]
            low[axis] -= 1
            lower = list(low)
            lower[axis] -= 1
            for n in range(L - s + 1):
                R[n, t, u, v] = D * R[(n + 1, *low)] + ((k - 1) * R[(n + 1, *lower)] if k > 1 else 0.0)
    return torch.stack([R[0, t, u, v] for t, u, v in triples(L)], dim=1)


class Plain:
    """Shells as 64-bit tensors: coefficients with the (L,0,0) primitive norm folded in, and every Cartesian
    component's normalisation to unit self-overlap."""

    def __init__(self, shells):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        K = max(len(s[2]) for s in shells)
        self.L = np.array([s[0] for s in shells])
        self.f0 = np.cumsum([0] + [(l + 1) * (l + 2) // 2 for l in self.L])
        ex, co, norm = np.ones((len(shells), K)), np.zeros((len(shells), K)), np.zeros((len(shells), 6))
        odd = lambda n: math.prod(range(n, 0, -2))  # noqa: E731
        for i, (L, _, e, c) in enumerate(shells):
            e = np.array(e)
            ex[i, :len(e)] = e
            co[i, :len(e)] = np.array(c) * np.sqrt((4 * e) ** L / ((math.pi / (2 * e)) ** 1.5 * odd(2 * L - 1)))
            p = ex[i][:, None] + ex[i][None, :]
            radial = float((co[i][:, None] * co[i][None, :] * (math.pi / p) ** 1.5 / (2 * p) ** L).sum())
            for k, m in enumerate(comps(L)):
                norm[i, k] = 1.0 / math.sqrt(radial * math.prod(odd(2 * x - 1) for x in m))
        as_t = lambda v: torch.tensor(v, dtype=torch.float64, device=self.dev)  # noqa: E731
        self.ex, self.co, self.norm, self.cen = as_t(ex), as_t(co), as_t(norm), as_t(np.array([s[1] for s in shells]))
        self.np = torch.tensor([len(s[2]) for s in shells], device=self.dev)

    def pair(self, a, i, b, j, la, lb):
        """primitive pairs: exponent sum, centre, prefactor, and the Hermite expansion of every component pair
        as [rows, na * nb, nherm(la + lb)]"""
        ea, eb, A, B = self.ex[a, i], self.ex[b, j], self.cen[a], self.cen[b]
        p = ea + eb
        P = (ea[:, None] * A + eb[:, None] * B) / p[:, None]
        K = self.co[a, i] * self.co[b, j] * torch.exp(-ea * eb / p * ((A - B) ** 2).sum(dim=1))
        E = [hermite(la, lb, P[:, x] - A[:, x], P[:, x] - B[:, x], p) for x in range(3)]
        H = triples(la + lb)
        where = {h: k for k, h in enumerate(H)}
        na, nb = comps(la), comps(lb)
        out = torch.zeros(len(a), len(na) * len(nb), len(H), dtype=torch.float64, device=self.dev)
        for ka, ca in enumerate(na):
            for kb, cb in enumerate(nb):
                ex, ey, ez = (E[x][ca[x]][cb[x]] for x in range(3))
                for t in range(len(ex)):
                    for u in range(len(ey)):
                        xy = ex[t] * ey[u]
                        for v in range(len(ez)):
                            out[:, ka * len(nb) + kb, where[t, u, v]] = xy * ez[v]
        return p, P, K, out

    def pair_norm(self, a, b, la, lb):
        na, nb = len(comps(la)), len(comps(lb))
        return (self.norm[a, :na, None] * self.norm[b, None, :nb]).reshape(len(a), na * nb)

    def eri(self, c, quartets):
        """(ab|cd) blocks of the quartets (n x 4 shell indices) of class c, [n, na * nb * nc * nd]"""
        la, lb, lc, ld = c
        q = torch.as_tensor(quartets, device=self.dev).long()
        hab, hcd = triples(la + lb), triples(lc + ld)
        where = {h: k for k, h in enumerate(triples(sum(c)))}
        index = torch.tensor([[where[tuple(x + y for x, y in zip(g, h))] for h in hcd] for g in hab], device=self.dev)
        sign = torch.tensor([(-1.0) ** sum(h) for h in hcd], dtype=torch.float64, device=self.dev)
        out = torch.zeros(len(q), block_size(c), dtype=torch.float64, device=self.dev)
        n = self.np[q]
        count = n.prod(dim=1)
        rows = torch.repeat_interleave(torch.arange(len(q), device=self.dev), count)
        x = torch.arange(len(rows), device=self.dev) - torch.repeat_interleave(count.cumsum(0) - count, count)
        step = max(256, int(4e8 / (8 * (len(hab) * len(hcd) + 3 * nherm(sum(c)) + block_size(c)))))
        for s in range(0, len(rows), step):
            r, k = rows[s:s + step], x[s:s + step]
            m = n[r]
            l, k = k % m[:, 3], k // m[:, 3]
            kk, k = k % m[:, 2], k // m[:, 2]
            j, i = k % m[:, 1], k // m[:, 1]
            p, P, Kab, Eab = self.pair(q[r, 0], i, q[r, 1], j, la, lb)
            g, Q, Kcd, Ecd = self.pair(q[r, 2], kk, q[r, 3], l, lc, ld)
            D = P - Q
            R = hermite_coulomb(sum(c), p * g / (p + g), D[:, 0], D[:, 1], D[:, 2])
            pre = 2.0 * math.pi ** 2.5 / (p * g * torch.sqrt(p + g)) * Kab * Kcd
            v = (Eab * pre[:, None, None]) @ R[:, index] @ (Ecd * sign).transpose(1, 2)
            out.index_add_(0, r, v.reshape(len(r), -1))
        return out * (self.pair_norm(q[:, 0], q[:, 1], la, lb)[:, :, None]
                      * self.pair_norm(q[:, 2], q[:, 3], lc, ld)[:, None, :]).reshape(len(q), -1)

    def pairs_of(self, x):
        a, b = np.tril_indices(len(self.L))
        a, b = np.where(self.L[a] >= self.L[b], a, b), np.where(self.L[a] >= self.L[b], b, a)
        keep = (self.L[a] == PAIRS[x][0]) & (self.L[b] == PAIRS[x][1])
        return a[keep], b[keep]

    def functions(self, shell, L):
        return torch.as_tensor(self.f0[:-1][shell], device=self.dev)[:, None] + torch.arange(len(comps(L)), device=self.dev)

    def eri_tensor(self):
        n = int(self.f0[-1])
        T = torch.zeros(n * n, n * n, dtype=torch.float64, device=self.dev)
        for X in range(6):
            for Y in range(X + 1):
                (a, b), (c, d) = self.pairs_of(X), self.pairs_of(Y)
                i, j = (v.reshape(-1) for v in np.meshgrid(np.arange(len(a)), np.arange(len(c)), indexing="ij"))
                if not len(i):
                    continue
                cls = PAIRS[X] + PAIRS[Y]
                v = self.eri(cls, np.stack([a[i], b[i], c[j], d[j]], axis=1)).reshape(len(i), block_size(PAIRS[X]), block_size(PAIRS[Y]))
                fa, fb, fc, fd = (self.functions(s, l) for s, l in zip((a[i], b[i], c[j], d[j]), cls))
                for u in (fa[:, :, None] * n + fb[:, None, :], fb[:, None, :] * n + fa[:, :, None]):
                    for w in (fc[:, :, None] * n + fd[:, None, :], fd[:, None, :] * n + fc[:, :, None]):
                        u2, w2 = u.reshape(len(i), -1, 1), w.reshape(len(i), 1, -1)
                        T[u2, w2] = v
                        T[w2, u2] = v
        return T.reshape(n, n, n, n)

    def one_electron(self, Z, R):
        """overlap and core Hamiltonian"""
        n = int(self.f0[-1])
        S, H = (torch.zeros(n, n, dtype=torch.float64, device=self.dev) for _ in range(2))
        Z, R = torch.tensor(Z, dtype=torch.float64, device=self.dev), torch.tensor(R, dtype=torch.float64, device=self.dev)
        for la in range(3):
            for lb in range(3):
                a, b = (v.reshape(-1) for v in np.meshgrid(np.flatnonzero(self.L == la), np.flatnonzero(self.L == lb), indexing="ij"))
                if not len(a):
                    continue
                a, b = torch.as_tensor(a, device=self.dev), torch.as_tensor(b, device=self.dev)
                na, nb = comps(la), comps(lb)
                s, h = (torch.zeros(len(a), len(na) * len(nb), dtype=torch.float64, device=self.dev) for _ in range(2))
                for i in range(int(self.np.max())):
                    for j in range(int(self.np.max())):
                        # absent primitives have coefficient zero
                        ia, jb = torch.full_like(a, i), torch.full_like(b, j)
                        p, P, K, E = self.pair(a, ia, b, jb, la, lb)
                        for z, c in zip(Z, R):
                            D = P - c
                            r = hermite_coulomb(la + lb, p, D[:, 0], D[:, 1], D[:, 2])
                            h -= (z * 2.0 * math.pi / p * K)[:, None] * (E @ r[:, :, None])[:, :, 0]
                        e = self.ex[b, jb]
                        W = [hermite(la, lb + 2, P[:, x] - self.cen[a, x], P[:, x] - self.cen[b, x], p) for x in range(3)]
                        w = K * (math.pi / p) ** 1.5
                        for ka, ca in enumerate(na):
                            for kb, cb in enumerate(nb):
                                o = [W[x][ca[x]][cb[x]][0] for x in range(3)]
                                # -1/2 d^2/dx^2 of x^m exp(-e x^2)
                                k2 = [e * (2 * cb[x] + 1) * o[x] - 2.0 * e * e * W[x][ca[x]][cb[x] + 2][0]
                                      - (0.5 * cb[x] * (cb[x] - 1) * W[x][ca[x]][cb[x] - 2][0] if cb[x] > 1 else 0.0) for x in range(3)]
                                s[:, ka * len(nb) + kb] += w * o[0] * o[1] * o[2]
                                h[:, ka * len(nb) + kb] += w * (k2[0] * o[1] * o[2] + o[0] * k2[1] * o[2] + o[0] * o[1] * k2[2])
                nrm = self.pair_norm(a, b, la, lb)
                fa, fb = self.functions(a.cpu().numpy(), la), self.functions(b.cpu().numpy(), lb)
                S[fa[:, :, None], fb[:, None, :]] = (s * nrm).reshape(len(a), len(na), len(nb))
                H[fa[:, :, None], fb[:, None, :]] = (h * nrm).reshape(len(a), len(na), len(nb))
        return S, H


def plain_rhf(kind, Z, R):
    """energy and total density of the closed-shell SCF, DIIS on the orthonormal-basis Fock matrix"""
    P = Plain(molecule_shells(kind, Z, R))
    S, H = (v.cpu().numpy() for v in P.one_electron(Z, R))
    n, occ = len(S), sum(Z) // 2
    T = P.eri_tensor()
    Jm = T.reshape(n * n, n * n)
    Km = T.permute(0, 2, 1, 3).reshape(n * n, n * n)
    nuc = sum(Z[i] * Z[j] / float(np.linalg.norm(R[i] - R[j])) for i in range(len(Z)) for j in range(i))
    w, U = np.linalg.eigh(S)
    X = U / np.sqrt(w)

    def occupied(F):
        _, C = np.linalg.eigh(F)
        C = X @ C[:, :occ]
        return 2.0 * C @ C.T

    D, kept = occupied(X.T @ H @ X), []
    for _ in range(200):
        d = torch.from_numpy(D).to(P.dev).reshape(-1)
        F = H + (Jm @ d - 0.5 * (Km @ d)).reshape(n, n).cpu().numpy()
        F = 0.5 * (F + F.T)
        energy = 0.5 * float((D * (H + F)).sum()) + nuc
        G = X.T @ F @ X
        err = X.T @ (F @ D @ S - S @ D @ F) @ X
        if np.linalg.norm(err) < 1e-9:
            break
        kept = (kept + [(G, err)])[-8:]
        m = len(kept)
        B = -np.ones((m + 1, m + 1))
        B[m, m] = 0.0
        B[:m, :m] = [[(x[1] * y[1]).sum() for y in kept] for x in kept]
        scale = max(1e-300, float(np.abs(B[:m, :m]).max()))
        B[:m, :m] /= scale
        c = np.linalg.lstsq(B, np.append(np.zeros(m), -1.0), rcond=None)[0][:m]
        D = occupied(sum(x * g[0] for x, g in zip(c, kept)))
    else:
        return None
    return energy, D


def exact(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind in ("eri", "eri_host"):
        if case["nq"] > 25000:
            return None
        plain = Plain(pool_shells(rng))
        return [plain.eri(c, q) for c, q in zip(CLASSES, pool_quartets(case["nq"], rng))]
    if kind == "jk":
        Z, R = cluster(case, rng)
        shells = molecule_shells(case["basis"], Z, R)
        n = nbf_of(shells)
        if n > JK_EXACT_NBF:
            return None
        D = density(n, 5 * case["waters"], seed)
        T = Plain(shells).eri_tensor()
        return torch.einsum("abcd,cd->ab", T, D), torch.einsum("abcd,bd->ac", T, D)
    if kind == "rhf":
        return plain_rhf(case["basis"], *molecules(case, seed)[0])
    if kind == "rhf_batch":
        if case["conformers"] > 8:
            return None
        r = [plain_rhf(case["basis"], Z, R) for Z, R in molecules(case, seed)]
        return None if None in r else np.array([x[0] for x in r])
    x, t, m, p = mlp_inputs(case, seed)
    p = [v.double().requires_grad_() for v in p]
    h = x.double()
    for k in range(0, len(p), 2):
        h = h @ p[k].T + p[k + 1]
        if k + 2 < len(p):
            h = torch.nn.functional.silu(h)
    loss = (m * (h - t.double()) ** 2).sum() / m.double().sum()
    grad = torch.autograd.grad(loss, p)
    return float(loss.detach()), torch.cat([g.reshape(-1) for g in grad])
