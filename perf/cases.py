"""Measured cases: the calls a program built on this framework spends its time in.

Every case goes through the package's Python entry points, the thin mirror of
the C ABI.  Kinds:

  fock    one two-electron build G = J - K/2 (FockEngine.fock_rhf on host
          arrays, or fock_rhf_device on device arrays): the call an RHF loop
          makes once per iteration; precision, engine and difference-density
          screening as the drivers set them
  uhf     the same for two spin densities (FockEngine.fock_uhf)
  jk      separate J and scaled K, as a hybrid-functional RKS driver asks
          for them (FockEngine.jk)
  scf     a whole molecule as the conformer evaluation runs it: one-electron
          integrals, engine, RHF to convergence on the device, teardown
  eri     contracted Cartesian blocks of listed shell quartets of one class
          (EriBatch.run), the class microbenchmark's call
  mp2     RMP2 correlation energy: dense AO tensor, four quarter transforms
          and the energy sum (FockEngine.rmp2_energy)
  predict forward pass of one learned-guess network (MLP.forward)
  train   minibatch training of one such network (MLP.train_step)
"""
import importlib
import math

import numpy as np
import torch

P = importlib.import_module("planck-refactored_b200")

BASES = ("sto-3g", "3-21g", "6-31g*", "6-31g**", "cc-pvdz")
PAIR_CLASSES = ((0, 0), (1, 0), (1, 1), (2, 0), (2, 1), (2, 2), (3, 0), (3, 1), (3, 2), (3, 3))
LETTERS = "spdf"
NFEAT, HIDDEN = 112, 256        # the learned-guess networks' input and hidden widths
EXACT_NBASIS = 130              # largest basis exact() works out


def listed():
    return [
        # a single small molecule: launches and host work decide
        {"name": "fock_water", "kind": "fock", "mol": "water", "n": 1, "basis": "6-31g**", "engine": "os",
         "precision": "fp64", "device": False, "tune": False, "screen": False},
        # the middle of the conformer sets (C8..C20), default options
        {"name": "fock_conformer14", "kind": "fock", "mol": "conformer", "n": 14, "basis": "6-31g*", "engine": "os",
         "precision": "fp64", "device": False, "tune": False, "screen": False},
        # the benchmark cluster, as the benchmark runs it
        {"name": "fock_cluster32_mixed", "kind": "fock", "mol": "water", "n": 32, "basis": "6-31g**",
         "engine": "auto", "precision": "mixed", "device": True, "tune": True, "screen": False},
        # the largest molecule: deep contractions, all FP64
        {"name": "fock_chain40", "kind": "fock", "mol": "alkane", "n": 40, "basis": "cc-pvdz", "engine": "auto",
         "precision": "fp64", "device": True, "tune": False, "screen": False},
        # a difference-density build between full builds: FP32 list, density screening
        {"name": "fock_difference20", "kind": "fock", "mol": "alkane", "n": 20, "basis": "cc-pvdz", "engine": "os",
         "precision": "mixed", "device": False, "tune": False, "screen": True},
        # open shell
        {"name": "uhf_water5", "kind": "uhf", "mol": "water", "n": 5, "basis": "6-31g**"},
        # J and scaled K of a hybrid functional
        {"name": "jk_pentane", "kind": "jk", "mol": "conformer", "n": 5, "basis": "cc-pvdz", "k_scale": 0.25},
        # a whole molecule from geometry to converged energy
        {"name": "scf_water4", "kind": "scf", "mol": "water", "n": 4, "basis": "6-31g**"},
        # integral blocks with an f shell
        {"name": "eri_fdpp", "kind": "eri", "bra": 8, "ket": 2, "n": 16384, "engine": "rys", "precision": "fp64"},
        # MP2 of a small cluster
        {"name": "mp2_water5", "kind": "mp2", "mol": "water", "n": 5, "basis": "6-31g**"},
        # the network of carbon pairs over the pairs of one molecule's conformers
        {"name": "predict_8192", "kind": "predict", "rows": 8192, "out": 232},
        # sixteen minibatches of its training
        {"name": "train_2048", "kind": "train", "rows": 2048, "out": 232, "steps": 16},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("fock", "fock", "fock", "uhf", "jk", "scf", "eri", "eri", "mp2", "predict", "train"))
    if kind in ("fock", "uhf", "jk"):
        mol = rng.choice(("water", "conformer", "alkane"))
        basis = rng.choice(BASES)
        top = {"water": 30, "conformer": 20, "alkane": 36}[mol]
        c = {"kind": kind, "mol": mol, "n": _log_int(rng, 1 if mol != "conformer" else 2, top), "basis": basis}
        if kind == "fock":
            mixed = rng.random() < 0.4
            c.update(engine=rng.choice(("os", "rys", "auto")), precision="mixed" if mixed else "fp64",
                     device=rng.random() < 0.5, tune=False, screen=mixed and rng.random() < 0.5)
        if kind == "jk":
            c["k_scale"] = rng.choice((0.2, 0.25, 1.0))
        if kind == "uhf":
            c["n"] = max(1, c["n"] // 2)
        return c
    if kind == "scf":
        return {"kind": "scf", "mol": "water", "n": _log_int(rng, 1, 8), "basis": rng.choice(("sto-3g", "6-31g**"))}
    if kind == "eri":
        bra = rng.randrange(10)
        ket = rng.randrange(bra + 1)
        ncomp = math.prod((l + 1) * (l + 2) // 2 for l in PAIR_CLASSES[bra] + PAIR_CLASSES[ket])
        top = max(1024, min(65536, 30_000_000 // ncomp))
        low = sum(PAIR_CLASSES[bra] + PAIR_CLASSES[ket]) <= 4
        return {"kind": "eri", "bra": bra, "ket": ket, "n": _log_int(rng, 33, top),
                "engine": rng.choice(("os", "rys")) if low else "rys", "precision": rng.choice(("fp64", "fp64", "mixed"))}
    if kind == "mp2":
        return {"kind": "mp2", "mol": "water", "n": rng.randint(1, 6), "basis": rng.choice(("sto-3g", "6-31g**"))}
    out = rng.choice((8, 16, 32, 64, 120, 232))
    if kind == "predict":
        return {"kind": "predict", "rows": _log_int(rng, 1, 8192), "out": out}
    return {"kind": "train", "rows": _log_int(rng, 64, 4096), "out": out, "steps": rng.randint(1, 16)}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
_LIB = P.basis.load_library()


def _atoms(case, seed):
    if case["mol"] == "water":
        return P.workloads.water_cluster(case["n"], seed=seed)
    if case["mol"] == "alkane":
        return P.workloads.alkane(case["n"], seed=seed)
    return P.workloads.alkane_conformer(case["n"], seed)


def _molecule(case, seed):
    return P.shells_for(_atoms(case, seed), case["basis"], _LIB)


def _ncart(l):
    return (int(l) + 1) * (int(l) + 2) // 2


def _density(shells, seed, scale=1.0):
    """A symmetric density with an insulator's decay: diagonal of order one,
    off-diagonal elements falling off over about two bond lengths."""
    centre = np.repeat(shells["center"], [_ncart(l) for l in shells["L"]], axis=0)
    nb = len(centre)
    x = torch.from_numpy(centre).cuda()
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randn((nb, nb), generator=g, device="cuda", dtype=torch.float64) * 0.3
    sq = (x * x).sum(1)
    r = (sq[:, None] + sq[None, :] - 2.0 * x @ x.T).clamp_min(0.0).sqrt()
    d = 0.5 * (a + a.T) * torch.exp(-r / 4.0)
    d += torch.diag(torch.rand(nb, generator=g, device="cuda", dtype=torch.float64) + 0.5)
    d = 0.5 * (d + d.T) * scale
    return d.cpu().numpy()


def _orbitals(shells, seed, nocc):
    """Orthonormal orbitals (columns over S) and separated orbital energies."""
    S = _overlap(shells)
    nb = S.shape[0]
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randn((nb, nb), generator=g, device="cuda", dtype=torch.float64)
    w, u = torch.linalg.eigh(S)
    x = u @ torch.diag(w.rsqrt()) @ u.T
    q, _ = torch.linalg.qr(a)
    eps = torch.rand(nb, generator=g, device="cuda", dtype=torch.float64)
    eps[:nocc] = -0.4 - 1.2 * eps[:nocc].sort(descending=True).values
    eps[nocc:] = 0.2 + 2.5 * eps[nocc:].sort().values
    return (x @ q).cpu().numpy(), eps.cpu().numpy()


def _features(rows, seed):
    """Radial Gaussians times direction cosines: values in [-1, 1], about half of them near zero."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = torch.rand((rows, NFEAT), generator=g, device="cuda")
    s = torch.rand((rows, NFEAT), generator=g, device="cuda") * 2.0 - 1.0
    return (torch.exp(-6.0 * r * r) * s).contiguous()


def _start_params(case, seed):
    return P.mlp.init_params(_dims(case), seed)


def _dims(case):
    return [NFEAT, HIDDEN, HIDDEN, case["out"]]


def _targets(case, X, seed):
    """Standardised outputs that depend on the inputs, with noise."""
    g = torch.Generator(device="cuda").manual_seed(seed + 7)
    W = torch.randn((NFEAT, case["out"]), generator=g, device="cuda") * 0.3
    n = torch.randn((X.shape[0], case["out"]), generator=g, device="cuda") * 0.3
    return (torch.tanh(X @ W) + n).contiguous()


def _batches(case, seed):
    out = []
    for k in range(case["steps"]):
        X = _features(case["rows"], 1000 * seed + k)
        out.append((X, _targets(case, X, seed)))
    return out


def _rates(case):
    """Cosine decay over the steps, as the training loop sets it."""
    return [1e-3 * 0.5 * (1.0 + math.cos(math.pi * k / case["steps"])) for k in range(case["steps"])]


def _quartets(case, seed):
    return P.workloads.eri_class_quartets(*PAIR_CLASSES[case["bra"]], *PAIR_CLASSES[case["ket"]], case["n"], seed=seed)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "eri":
        shells, pairs, quartets = _quartets(case, seed)
        b = P.EriBatch(shells, pairs, quartets)
        out = torch.empty((b.n, b.ncomp), dtype=torch.float64, device="cuda")
        return {"case": case, "batch": b, "out": out, "stream": torch.cuda.Stream()}
    if kind == "predict":
        net = P.mlp.MLP(_dims(case), max(case["rows"], 8), params=_start_params(case, seed))
        return {"case": case, "net": net, "X": _features(case["rows"], seed)}
    if kind == "train":
        p0 = _start_params(case, seed)
        net = P.mlp.MLP(_dims(case), case["rows"], params=p0)
        return {"case": case, "net": net, "p0": p0, "batches": _batches(case, seed), "rates": _rates(case)}
    if kind == "scf":
        return {"case": case, "atoms": _atoms(case, seed)}
    mol, shells = _molecule(case, seed)
    if kind == "mp2":
        nocc = mol.nelectron() // 2
        C, eps = _orbitals(shells, seed, nocc)
        return {"case": case, "engine": P.FockEngine(shells), "C": C, "eps": eps, "nocc": nocc}
    if kind == "uhf":
        return {"case": case, "engine": P.FockEngine(shells), "Pa": _density(shells, seed, 0.5),
                "Pb": _density(shells, seed + 1, 0.5)}
    if kind == "jk":
        return {"case": case, "engine": P.FockEngine(shells), "P": _density(shells, seed)}
    screen = case["screen"]
    # difference builds: every quartet on the FP32 list, as the incremental driver sets it
    eng = P.FockEngine(shells, engine=case["engine"], precision=case["precision"],
                       fp32_bound=1e300 if screen else 1e-8)
    if screen:
        eng.set_density_screening(1e-12)
    if case["tune"]:
        eng.autotune()
    D = _density(shells, seed, 1e-5 if screen else 1.0)
    st = {"case": case, "engine": eng, "P": D}
    if case["device"]:
        st.update(dP=torch.from_numpy(D).cuda(), dG=torch.zeros(D.shape, dtype=torch.float64, device="cuda"),
                  stream=torch.cuda.Stream())
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "fock":
        if not case["device"]:
            return st["engine"].fock_rhf(st["P"])
        st["engine"].fock_rhf_device(st["dP"].data_ptr(), st["dG"].data_ptr(), st["stream"].cuda_stream)
        return st["dG"]
    if kind == "uhf":
        return st["engine"].fock_uhf(st["Pa"], st["Pb"])
    if kind == "jk":
        return st["engine"].jk(st["P"], k_scale=case["k_scale"])
    if kind == "scf":
        s = P.scf.System(st["atoms"], case["basis"], _LIB)
        r = s.run(linalg="gpu")
        s.close()
        return {"energy": r["energy"], "P": r["P"], "eps": r["eps"], "S": s.S, "H": s.H}
    if kind == "eri":
        st["batch"].run(0, st["batch"].n, case["engine"], case["precision"], st["out"].data_ptr(),
                        st["stream"].cuda_stream)
        return st["out"]
    if kind == "mp2":
        return st["engine"].rmp2_energy(st["C"], st["eps"], st["nocc"])
    if kind == "predict":
        return st["net"].forward(st["X"])
    st["net"].set_params(st["p0"])
    losses = [st["net"].train_step(X, T, lr) for (X, T), lr in zip(st["batches"], st["rates"])]
    return {"losses": np.array(losses), "params": st["net"].params()}


# ---------------------------------------------------------------------------
# Work and tolerance
# ---------------------------------------------------------------------------
def _class_flops(bra, ket, prims):
    """FP64 work of `prims` primitive quartets of a class by Rys quadrature."""
    (la, lb), (lc, ld) = bra, ket
    e, f = la + lb, lc + ld
    nr = (e + f) // 2 + 1
    N = _ncart(la) * _ncart(lb) * _ncart(lc) * _ncart(ld)
    return prims * (nr * (12 * (e + 1) * (f + 1) + 6 * (la + 1) * (lb + 1) * (lc + 1) * (ld + 1) + 3 * N) + 40)


def _fock_flops(shells):
    """Primitive quartets of the shell quartets that pass Q Q >= 1e-10, with
    Q estimated from each pair's widest primitives, times the class's work.
    Only primitive pairs whose Gaussian product is above 1e-16 count, and
    shells of one centre that share their exponents (general contractions)
    count their primitives once between them."""
    L, npr, R = shells["L"], shells["nprim"], shells["center"]
    ns = len(L)
    off = np.concatenate([[0], np.cumsum(npr)])
    amin = np.array([shells["expo"][off[s]:off[s + 1]].min() for s in range(ns)])
    key = [(int(L[s]), *R[s], *shells["expo"][off[s]:off[s + 1]]) for s in range(ns)]
    count = {}
    for k in key:
        count[k] = count.get(k, 0) + 1
    share = np.array([1.0 / count[k] for k in key])
    of = np.repeat(np.arange(ns), npr)
    i, j = np.triu_indices(ns)
    K = np.zeros((ns, ns))
    r2 = ((R[:, None, :] - R[None, :, :]) ** 2).sum(-1)
    for s in range(ns):
        for e in shells["expo"][off[s]:off[s + 1]]:
            live = e * shells["expo"] / (e + shells["expo"]) * r2[s][of] < 37.0
            K[s] += np.bincount(of[live], minlength=ns)
    K *= share[:, None] * share[None, :]
    K = K[i, j]
    z = amin[i] + amin[j]
    q = np.exp(-amin[i] * amin[j] / z * r2[i, j]) * (amin[i] * amin[j] / z ** 2) ** 0.75 * z ** 0.25 * 1.1
    pc = np.maximum(L[i], L[j]) * (np.maximum(L[i], L[j]) + 1) // 2 + np.minimum(L[i], L[j])
    total = 0.0
    by = {}
    for x in range(10):
        m = pc == x
        if m.any():
            o = np.argsort(-q[m], kind="stable")
            by[x] = (q[m][o], K[m][o])
    for x, (qx, kx) in by.items():
        for y, (qy, ky) in by.items():
            if y > x:
                continue
            n = np.searchsorted(-qy, -1e-10 / qx, side="right")
            prims = float((kx * np.concatenate([[0.0], np.cumsum(ky)])[n]).sum()) * (0.5 if x == y else 1.0)
            total += _class_flops(PAIR_CLASSES[x], PAIR_CLASSES[y], prims)
    return total


def work(case):
    kind = case["kind"]
    if kind in ("predict", "train"):
        d = _dims(case)
        macs = sum(a * b for a, b in zip(d[:-1], d[1:]))
        params = macs + sum(d[1:])
        if kind == "predict":
            return {"bytes": 4.0 * (case["rows"] * (d[0] + d[-1]) + params), "flops": 2.0 * case["rows"] * macs}
        # forward, weight gradients, and input gradients of all layers but the first
        flops = 2.0 * case["rows"] * (3 * macs - d[0] * d[1])
        # the batch, and parameters and both moments read and written
        return {"bytes": case["steps"] * 4.0 * (case["rows"] * (d[0] + d[-1]) + 6 * params), "flops": case["steps"] * flops}
    if kind == "eri":
        bra, ket = PAIR_CLASSES[case["bra"]], PAIR_CLASSES[case["ket"]]
        ncomp = math.prod(_ncart(l) for l in bra + ket)
        prims = case["n"] * 3.5 ** 4            # contraction depths uniform in 1..6
        return {"bytes": case["n"] * (8.0 * ncomp + 2 * 12.25 * 80), "flops": _class_flops(bra, ket, prims)}
    mol, shells = _molecule(case, 1)
    nb = sum(_ncart(l) for l in shells["L"])
    f = _fock_flops(shells)
    if kind == "fock":
        return {"bytes": 16.0 * nb * nb, "flops": f}
    if kind == "uhf":
        return {"bytes": 32.0 * nb * nb, "flops": f}
    if kind == "jk":
        return {"bytes": 24.0 * nb * nb, "flops": f}
    if kind == "mp2":
        o = mol.nelectron() // 2
        v = nb - o
        quarter = 2.0 * (nb ** 4 * o + nb ** 3 * o * v + nb ** 2 * o * v * o + nb * o * v * o * v)
        return {"bytes": 8.0 * (nb * nb + nb), "flops": f + quarter}
    # about fifteen iterations of one build and six products and an eigensolution of about nine more
    return {"bytes": 8.0 * 4 * nb * nb, "flops": 15 * (f + 15 * 2.0 * nb ** 3)}


def tolerance(case):
    """About four times the largest error seen against exact(), or against
    another engine where the Schwarz screen (1e-10 on integrals, part of the
    definition of the result) would dominate that."""
    kind = case["kind"]
    if kind == "predict":
        return {"rel": 1.6e-2, "max": 1e-1}     # BF16 products, FP32 sums
    if kind == "train":
        return {"rel": 2e-3}
    if kind == "scf":
        return {"rel": 1e-8}                    # converged to 1e-10 in the density
    if kind == "eri":
        return {"rel": 1e-4} if case["precision"] == "mixed" else {"rel": 1e-11}
    if kind == "fock" and case["precision"] == "mixed":
        return {"rel": 1e-5} if case["screen"] else {"rel": 1e-10}
    return {"rel": 1e-11}


# ---------------------------------------------------------------------------
# The same quantities in plain 64-bit torch: McMurchie-Davidson integrals
# ---------------------------------------------------------------------------
F64 = dict(dtype=torch.float64, device="cuda")


def _cart(l):
    return [(x, y, l - x - y) for x in range(l, -1, -1) for y in range(l - x, -1, -1)]


def _dfact(n):
    return 1.0 if n <= 1 else n * _dfact(n - 2)


def _cnorm(l):
    return torch.tensor([1.0 / math.sqrt(_dfact(2 * x - 1) * _dfact(2 * y - 1) * _dfact(2 * z - 1))
                         for x, y, z in _cart(l)], **F64)


def _hermites(n):
    return [(t, u, v) for s in range(n + 1) for t in range(s, -1, -1) for u in range(s - t, -1, -1) for v in (s - t - u,)]


def _expansion(la, lb, PA, PB, z):
    """1-D Hermite expansion coefficients E[i][j][t] without the Gaussian factor; PA, PB, z of one shape."""
    one, zero = torch.ones_like(z), torch.zeros_like(z)
    E = {(0, 0): [one]}

    def get(i, j, t):
        e = E[(i, j)]
        return e[t] if 0 <= t < len(e) else zero

    for i in range(la + 1):
        for j in range(lb + 1):
            if (i, j) == (0, 0):
                continue
            s, X = ((i - 1, j), PA) if i > 0 else ((i, j - 1), PB)
            E[(i, j)] = [get(*s, t - 1) / (2.0 * z) + X * get(*s, t) + (t + 1) * get(*s, t + 1) for t in range(i + j + 1)]
    return E


def _boys(M, T):
    """F_0 .. F_M: series and downward recurrence below 40, the large-T limit above."""
    Ts = T.clamp(max=40.0)
    e = torch.exp(-Ts)
    term = torch.ones_like(Ts) / (2 * M + 1)
    s = term.clone()
    for k in range(1, 160):
        term = term * (2.0 * Ts / (2 * M + 2 * k + 1))
        s += term
    F = [None] * (M + 1)
    F[M] = e * s
    for m in range(M - 1, -1, -1):
        F[m] = (2.0 * Ts * F[m + 1] + e) / (2 * m + 1)
    big = T > 40.0
    Tb = T.clamp(min=1.0)
    g = 0.5 * torch.sqrt(math.pi / Tb)
    for m in range(M + 1):
        F[m] = torch.where(big, g, F[m])
        g = g * (2 * m + 1) / (2.0 * Tb) - torch.exp(-Tb) / (2.0 * Tb)
    return F


def _hermite_coulomb(L, a, X):
    """R_tuv, t + u + v <= L, stacked in the order of _hermites(L); a and X (..., 3) broadcast."""
    T = a * (X * X).sum(-1)
    F = _boys(L, T)
    R = {(0, 0, 0): [((-2.0 * a) ** m) * F[m] for m in range(L + 1)]}
    for t, u, v in _hermites(L)[1:]:
        d = 0 if t else 1 if u else 2
        low = [t, u, v]
        low[d] -= 1
        p = R[tuple(low)]
        n = L - (t + u + v)
        x = [X[..., d] * p[m + 1] for m in range(n + 1)]
        if low[d] > 0:
            low2 = list(low)
            low2[d] -= 1
            pp = R[tuple(low2)]
            x = [x[m] + low[d] * pp[m + 1] for m in range(n + 1)]
        R[(t, u, v)] = x
    return torch.stack([R[h][0] for h in _hermites(L)], -1)


class _Pairs:
    """Shell pairs of one (la, lb), primitive pairs padded to one count."""

    def __init__(self, shells, ab, la, lb):
        off = np.concatenate([[0], np.cumsum(shells["nprim"])])
        ab = np.asarray(ab).reshape(-1, 2)
        n = len(ab)
        K = int(max(shells["nprim"][a] * shells["nprim"][b] for a, b in ab))
        al, be, cf = np.ones((n, K)), np.ones((n, K)), np.zeros((n, K))
        for p, (a, b) in enumerate(ab):
            sa, sb = slice(off[a], off[a + 1]), slice(off[b], off[b + 1])
            ea, eb = shells["expo"][sa], shells["expo"][sb]
            c = np.multiply.outer((shells["coef"] * shells["norm"])[sa], (shells["coef"] * shells["norm"])[sb]).ravel()
            k = len(c)
            al[p, :k], be[p, :k], cf[p, :k] = np.repeat(ea, len(eb)), np.tile(eb, len(ea)), c
        self.la, self.lb, self.n, self.K = la, lb, n, K
        al, be, cf = (torch.tensor(x, **F64) for x in (al, be, cf))
        A = torch.tensor(shells["center"][ab[:, 0]], **F64)[:, None, :]
        B = torch.tensor(shells["center"][ab[:, 1]], **F64)[:, None, :]
        z = al + be
        self.z = z
        self.P = (al[..., None] * A + be[..., None] * B) / z[..., None]
        kab = cf * torch.exp(-al * be / z * ((A - B) ** 2).sum(-1))
        self.be, self.kab = be, kab
        self.E1 = [_expansion(la, lb + 2, self.P[..., d] - A[..., d], self.P[..., d] - B[..., d], z) for d in range(3)]
        self.herm = _hermites(la + lb)
        self.norm = (_cnorm(la)[:, None] * _cnorm(lb)[None, :]).reshape(-1)
        rows = []
        for ca in _cart(la):
            for cb in _cart(lb):
                e = [self.E1[d][(ca[d], cb[d])] for d in range(3)]
                rows.append(torch.stack([e[0][t] * e[1][u] * e[2][v] if t < len(e[0]) and u < len(e[1]) and v < len(e[2])
                                         else torch.zeros_like(z) for t, u, v in self.herm], -1) * kab[..., None])
        # (n, K, comps, herm), component norms included
        self.E = torch.stack(rows, -2) * self.norm[:, None]


def _contract(bra, ket, X, pairwise):
    """(bra|ket) blocks, (nb, nk, AB, CD), or (n, AB, CD) when pairwise."""
    L = bra.la + bra.lb + ket.la + ket.lb
    index = {h: i for i, h in enumerate(_hermites(L))}
    idx = torch.tensor([[index[tuple(a + b for a, b in zip(h, g))] for g in ket.herm] for h in bra.herm], device="cuda")
    sign = torch.tensor([(-1.0) ** sum(g) for g in ket.herm], **F64)
    bs, ks = X
    zb, Pb, Eb = bra.z[bs], bra.P[bs], bra.E[bs]
    zk, Pk, Ek = ket.z[ks], ket.P[ks], ket.E[ks] * sign
    if pairwise:
        zb, zk, Pb, Pk = zb[:, :, None], zk[:, None, :], Pb[:, :, None, :], Pk[:, None, :, :]
    else:
        zb, zk, Pb, Pk = zb[:, None, :, None], zk[None, :, None, :], Pb[:, None, :, None, :], Pk[None, :, None, :, :]
    a = zb * zk / (zb + zk)
    R = _hermite_coulomb(L, a, Pb - Pk) * (2.0 * math.pi ** 2.5 / (zb * zk * torch.sqrt(zb + zk)))[..., None]
    G = R[..., idx]          # (..., Kb, Kk, hb, hk)
    if pairwise:
        return torch.einsum("npah,npqhg,nqcg->nac", Eb, G, Ek) if G.shape[1] * G.shape[2] == 1 else torch.einsum(
            "npah,nphc->nac", Eb, torch.einsum("npqhg,nqcg->nphc", G, Ek))
    return torch.einsum("bpah,bkphc->bkac", Eb, torch.einsum("bkpqhg,kqcg->bkphc", G, Ek))


def _ao_offsets(shells):
    n = [_ncart(l) for l in shells["L"]]
    return np.concatenate([[0], np.cumsum(n)])


def _pair_groups(shells):
    """Shell pairs by (la, lb, primitive pairs), la >= lb."""
    groups = {}
    for a in range(len(shells["L"])):
        for b in range(a, len(shells["L"])):
            x, y = (a, b) if shells["L"][a] >= shells["L"][b] else (b, a)
            key = (int(shells["L"][x]), int(shells["L"][y]), int(shells["nprim"][x] * shells["nprim"][y]))
            groups.setdefault(key, []).append((x, y))
    return [(k, np.array(v)) for k, v in sorted(groups.items())]


def _tensor(shells):
    """All (ij|kl), nb^4."""
    off = _ao_offsets(shells)
    nb = int(off[-1])
    T = torch.zeros((nb, nb, nb, nb), **F64)
    groups = [( _Pairs(shells, ab, la, lb), ab) for (la, lb, _), ab in _pair_groups(shells)]

    def functions(p, ab, rows):
        na, nbb = _ncart(p.la), _ncart(p.lb)
        i = torch.tensor(off[ab[rows, 0]], device="cuda")[:, None] + torch.arange(na, device="cuda").repeat_interleave(nbb)
        j = torch.tensor(off[ab[rows, 1]], device="cuda")[:, None] + torch.arange(nbb, device="cuda").repeat(na)
        return i, j

    for x, (pb, ab) in enumerate(groups):
        for pk, cd in groups[:x + 1]:
            per = pb.K * pk.K * len(pb.herm) * len(pk.herm) * 3 + pb.K * pk.K * 200
            nk = max(1, min(pk.n, 200_000_000 // (per * min(pb.n, 16))))
            nr = max(1, min(pb.n, 200_000_000 // (per * nk)))
            for b0 in range(0, pb.n, nr):
                for k0 in range(0, pk.n, nk):
                    bs, ks = np.arange(b0, min(pb.n, b0 + nr)), np.arange(k0, min(pk.n, k0 + nk))
                    v = _contract(pb, pk, (bs, ks), False)
                    i, j = functions(pb, ab, bs)
                    k, l = functions(pk, cd, ks)
                    i, j = i[:, None, :, None], j[:, None, :, None]
                    k, l = k[None, :, None, :], l[None, :, None, :]
                    for p, q in ((i, j), (j, i)):
                        for r, s in ((k, l), (l, k)):
                            T[p, q, r, s] = v
                            T[r, s, p, q] = v
    return T


def _overlap(shells):
    return _one_electron(shells, None)[0]


def _one_electron(shells, nuclei):
    """S, T and V (None without nuclei)."""
    off = _ao_offsets(shells)
    nb = int(off[-1])
    out = [torch.zeros((nb, nb), **F64) for _ in range(3)]
    for (la, lb, _), ab in _pair_groups(shells):
        p = _Pairs(shells, ab, la, lb)
        root = (math.pi / p.z).sqrt()
        E0 = [[[p.E1[d][(i, j)][0] * root for j in range(lb + 3)] for i in range(la + 1)] for d in range(3)]

        def kin(d, i, j):
            t = 4.0 * p.be ** 2 * E0[d][i][j + 2] - 2.0 * p.be * (2 * j + 1) * E0[d][i][j]
            if j >= 2:
                t = t + j * (j - 1) * E0[d][i][j - 2]
            return -0.5 * t

        s, t = [], []
        for ca in _cart(la):
            for cb in _cart(lb):
                o = [E0[d][ca[d]][cb[d]] for d in range(3)]
                k = [kin(d, ca[d], cb[d]) for d in range(3)]
                s.append((p.kab * o[0] * o[1] * o[2]).sum(1))
                t.append((p.kab * (k[0] * o[1] * o[2] + o[0] * k[1] * o[2] + o[0] * o[1] * k[2])).sum(1))
        vals = [torch.stack(s, -1) * p.norm, torch.stack(t, -1) * p.norm]
        if nuclei is not None:
            v = torch.zeros((p.n, len(s)), **F64)
            for x, y, zc, q in nuclei:
                R = _hermite_coulomb(la + lb, p.z, p.P - torch.tensor([x, y, zc], **F64))
                v -= q * torch.einsum("nkch,nkh->nc", p.E, R * (2.0 * math.pi / p.z)[..., None])
            vals.append(v)
        na, nbb = _ncart(la), _ncart(lb)
        i = torch.tensor(off[ab[:, 0]], device="cuda")[:, None] + torch.arange(na, device="cuda").repeat_interleave(nbb)
        j = torch.tensor(off[ab[:, 1]], device="cuda")[:, None] + torch.arange(nbb, device="cuda").repeat(na)
        for m, v in zip(out, vals):
            m[i, j] = v
            m[j, i] = v
    return out[0], out[1], out[2] if nuclei is not None else None


def _exact_jk(T, D):
    D = torch.tensor(D, **F64)
    return torch.einsum("ijkl,kl->ij", T, D), torch.einsum("ikjl,kl->ij", T, D)


def _exact_scf(case, seed):
    atoms = _atoms(case, seed)
    mol, shells = P.shells_for(atoms, case["basis"], _LIB)
    nuc = [(*map(float, x), float(z)) for x, z in zip(mol.coords, mol.Z)]
    S, T, V = _one_electron(shells, nuc)
    H = T + V
    X4 = _tensor(shells)
    enuc = sum(nuc[a][3] * nuc[b][3] / math.dist(nuc[a][:3], nuc[b][:3]) for a in range(len(nuc)) for b in range(a))
    nocc = mol.nelectron() // 2
    w, u = torch.linalg.eigh(S)
    X = u @ torch.diag(w.rsqrt()) @ u.T

    def density(F):
        eps, c = torch.linalg.eigh(X.T @ F @ X)
        c = X @ c
        return eps, 2.0 * c[:, :nocc] @ c[:, :nocc].T

    _, D = density(H)
    Fs, Es = [], []
    for _ in range(100):
        J, K = _exact_jk(X4, D)
        F = H + J - 0.5 * K
        E = 0.5 * float((D * (H + F)).sum()) + enuc
        err = X.T @ (F @ D @ S - S @ D @ F) @ X
        Fs, Es = (Fs + [F])[-8:], (Es + [err])[-8:]
        m = len(Fs)
        Fx = F
        if m > 1:
            B = torch.zeros((m + 1, m + 1), **F64)
            B[:m, :m] = torch.tensor([[float((a * b).sum()) for b in Es] for a in Es], **F64)
            B[:m, m] = B[m, :m] = -1.0
            rhs = torch.zeros(m + 1, **F64)
            rhs[m] = -1.0
            c = torch.linalg.pinv(B, rtol=1e-15) @ rhs
            Fx = sum(c[k] * Fs[k] for k in range(m))
        eps, Dn = density(Fx)
        step = float((Dn - D).abs().max())
        D = Dn
        if step < 1e-11:
            break
    return {"energy": E, "P": D, "eps": eps, "S": S, "H": H}


def _exact_eri(case, seed):
    shells, pairs, quartets = _quartets(case, seed)
    n = case["n"]
    bra = _Pairs(shells, pairs[0::2], *PAIR_CLASSES[case["bra"]])
    ket = _Pairs(shells, pairs[1::2], *PAIR_CLASSES[case["ket"]])
    per = bra.K * ket.K * (len(bra.herm) * len(ket.herm) * 3 + 400)
    step = max(1, 400_000_000 // per)
    out = [_contract(bra, ket, (np.arange(k, min(n, k + step)),) * 2, True) for k in range(0, n, step)]
    return torch.cat(out).reshape(n, -1)


def _exact_net(case, params, X):
    acts, zs, o = [X.double()], [], 0
    d = _dims(case)
    for k, (a, b) in enumerate(zip(d[:-1], d[1:])):
        W, bias = params[o:o + a * b].view(a, b), params[o + a * b:o + a * b + b]
        o += a * b + b
        zs.append(acts[-1] @ W + bias)
        acts.append(zs[-1] if k == len(d) - 2 else torch.nn.functional.silu(zs[-1]))
    return acts[-1]


def _exact_train(case, seed):
    p = torch.tensor(_start_params(case, seed), **F64)
    m, v, losses = torch.zeros_like(p), torch.zeros_like(p), []
    for k, ((X, T), lr) in enumerate(zip(_batches(case, seed), _rates(case)), 1):
        q = p.clone().requires_grad_(True)
        loss = ((_exact_net(case, q, X) - T.double()) ** 2).mean()
        g, = torch.autograd.grad(loss, q)
        m = 0.9 * m + 0.1 * g
        v = 0.999 * v + 0.001 * g * g
        p = p - lr * (m / (1 - 0.9 ** k)) / ((v / (1 - 0.999 ** k)).sqrt() + 1e-8)
        losses.append(float(loss))
    return {"losses": np.array(losses), "params": p}


def exact(case, seed):
    kind = case["kind"]
    if kind == "predict":
        with torch.no_grad():
            return _exact_net(case, torch.tensor(_start_params(case, seed), **F64), _features(case["rows"], seed))
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "eri":
        L = sum(PAIR_CLASSES[case["bra"]] + PAIR_CLASSES[case["ket"]])
        return _exact_eri(case, seed) if L <= 8 else None
    mol, shells = _molecule(case, seed)
    if sum(_ncart(l) for l in shells["L"]) > EXACT_NBASIS:
        return None
    if kind == "scf":
        return _exact_scf(case, seed)
    T = _tensor(shells)
    if kind == "mp2":
        nocc = mol.nelectron() // 2
        C, eps = (torch.tensor(x, **F64) for x in _orbitals(shells, seed, nocc))
        o, v = C[:, :nocc], C[:, nocc:]
        T = torch.einsum("ijkl,ia->ajkl", T, o)
        T = torch.einsum("ajkl,jb->abkl", T, v)
        T = torch.einsum("abkl,kc->abcl", T, o)
        T = torch.einsum("abcl,ld->abcd", T, v)
        e, w = eps[:nocc], eps[nocc:]
        den = e[:, None, None, None] + e[None, None, :, None] - w[None, :, None, None] - w[None, None, None, :]
        return float((T * (2.0 * T - T.permute(0, 3, 2, 1)) / den).sum())
    if kind == "uhf":
        Pa, Pb = _density(shells, seed, 0.5), _density(shells, seed + 1, 0.5)
        (Ja, Ka), (Jb, Kb) = _exact_jk(T, Pa), _exact_jk(T, Pb)
        return Ja + Jb - Ka, Ja + Jb - Kb
    if kind == "jk":
        J, K = _exact_jk(T, _density(shells, seed))
        return J, case["k_scale"] * K
    J, K = _exact_jk(T, _density(shells, seed, 1e-5 if case["screen"] else 1.0))
    return J - 0.5 * K
