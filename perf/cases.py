"""Timed cases of the integral engine, through its public Python entry points.

A case is a molecule, the call a program makes on it and the options it sets:

* ``mol``   the molecule: "water0" is the minimal-basis water, "water" a
            cluster of ``size`` waters in a def2-SVP-like basis, "organic" the
            ``size`` innermost atoms of the 24-atom organic molecule (s, p, d
            shells, contractions up to 6), "highl" the ``size`` innermost atoms
            of the 60-atom molecule with f shells (contractions up to 8),
            "batch" ``size`` small molecules of 3 to 30 atoms.
* ``call``  "g": build_rhf_g on host arrays; "j": build_coulomb_j on host
            arrays (pure density functionals); "jk": J and K on host arrays;
            "graph": J and K on device buffers, the whole build one CUDA graph
            replayed per step; "incremental": dP update and read-back of G;
            "onee": overlap, kinetic and nuclear-attraction matrices.
* ``tau``   Schwarz threshold; ``mixed`` the FP32/FP64 split threshold
            (0: plain FP64 build); ``den`` the density (CVHF) threshold.

A program keeps the basis, the plan, its buffers and the captured graph across
the steps of an SCF run, so ``prepare`` makes those and a density.
"""
import math

import numpy as np
import torch

from origo_tlno_b200 import engine as E
from origo_tlno_b200 import molecules as MOL

F64 = torch.float64


def _case(name, mol, size, call, tau, mixed=0.0, den=0.0):
    return {"name": name, "mol": mol, "size": size, "call": call, "tau": tau, "mixed": mixed, "den": den}


def listed():
    return [
        # a single small molecule in a minimal basis: launch count and latency
        _case("water-minimal-g", "water0", 1, "g", 1e-12),
        # a water dimer per SCF step from a captured graph: latency of one replay
        _case("water2-graph", "water", 2, "graph", 1e-12),
        # the ordinary job of a quantum-chemistry program: one organic molecule, host arrays
        _case("organic24-jk", "organic", 24, "jk", 1e-12),
        # a solvated fragment, mixed precision, all on the device
        _case("organic17-mixed-graph", "organic", 17, "graph", 1e-11, mixed=1e-7),
        # a small cluster in a long SCF run: density-difference updates
        _case("water12-incremental", "water", 12, "incremental", 1e-11, den=1e-11),
        # Coulomb matrix alone, as a pure functional needs it
        _case("water30-j", "water", 30, "j", 1e-11),
        # ordinary clusters, plain and mixed precision
        _case("water40-graph", "water", 40, "graph", 1e-11),
        _case("water91-mixed-graph", "water", 91, "graph", 1e-11, mixed=1e-7),
        # the largest build here
        _case("water160-graph", "water", 160, "graph", 1e-11),
        # f shells and deep contractions
        _case("highl14-graph", "highl", 14, "graph", 1e-12),
        # many small molecules at once (conformer or data-set generation)
        _case("batch48-graph", "batch", 48, "graph", 1e-12),
        # one-electron matrices of a new geometry
        _case("water50-onee", "water", 50, "onee", 1e-11),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    mol = rng.choice(["water", "water", "water", "organic", "organic", "highl", "batch"])
    tau = rng.choice([1e-10, 1e-11, 1e-12])
    mixed = den = 0.0
    if mol == "batch":
        size, call = _log_int(rng, 6, 48), "graph"
    elif mol == "highl":
        size, call = rng.randint(3, 14), rng.choice(["graph", "jk", "g"])
    elif mol == "organic":
        size, call = rng.randint(3, 24), rng.choice(["graph", "graph", "jk", "g", "incremental"])
    else:
        size = _log_int(rng, 1, 120)
        call = rng.choice(["graph", "graph", "graph", "jk", "g", "j", "incremental", "onee"])
    if call == "graph" and mol != "batch" and rng.random() < 0.4:
        mixed = rng.choice([1e-7, 1e-8, 1e-9])
    if call == "incremental":
        tau, den = max(tau, 1e-11), rng.choice([1e-10, 1e-11])
    return {"mol": mol, "size": size, "call": call, "tau": tau, "mixed": mixed, "den": den}


def _innermost(mol, n):
    """The n atoms of a molecule nearest to the centre of its atoms."""
    d = np.linalg.norm(mol.coords - mol.coords.mean(axis=0), axis=1)
    return MOL.fragment(mol, sorted(np.argsort(d, kind="stable")[:n]))


def _molecules(case):
    kind, n = case["mol"], case["size"]
    if kind == "water0":
        return [MOL.cfg0()]
    if kind == "water":
        # n waters on a near-cubic grid with about a tenth of its sites empty
        side = max(1, math.ceil((n * 1.12) ** (1.0 / 3.0)))
        nx = max(1, math.ceil(n * 1.12 / (side * side)))
        return [MOL.water_cluster(n, seed=5, grid=(nx, side, side))]
    if kind == "organic":
        return [_innermost(MOL.cfg1(), n)]
    if kind == "highl":
        return [_innermost(MOL.cfg2(), n)]
    return MOL.cfg3(n)


def _density(n_bf, seed, scale=1.0):
    """scale * C C^T, C (n_bf x n_bf/5) ~ N(0,1)/sqrt(n_bf), exactly symmetric."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    c = torch.randn(n_bf, max(1, n_bf // 5), generator=g, device="cuda", dtype=F64) / math.sqrt(n_bf)
    d = scale * (c @ c.T)
    return 0.5 * (d + d.T)


def _options(case):
    return E.ScreeningOptions(integral_threshold=case["tau"],
                              mixed_threshold=case["mixed"] if case["mixed"] > 0.0 else 1e-9)


def prepare(case, seed):
    mols, call, opts = _molecules(case), case["call"], _options(case)
    if call == "onee":
        # the geometry is the input: every seed moves the atoms a little
        mol = mols[0]
        shift = np.random.default_rng(seed).normal(scale=0.02, size=mol.coords.shape)
        return {"call": call, "mol": _moved(mol, shift), "plan": E.build_one_electron_plan(_moved(mol, shift))}
    contexts = [E.Context(m) for m in mols]
    if case["mol"] == "batch":
        b = E.Batch(contexts, opts)
        d = torch.cat([_density(c.M, seed + 7919 * k).reshape(-1) for k, c in enumerate(contexts)])
        j, k = torch.empty_like(d), torch.empty_like(d)
        torch.cuda.synchronize()
        b.graph_capture(d.data_ptr(), j.data_ptr(), k.data_ptr())
        return {"call": call, "handle": b, "stream": torch.cuda.ExternalStream(b.stream()), "d": d, "j": j, "k": k}
    ctx = contexts[0].plan(opts)
    if call == "graph":
        d = _density(ctx.M, seed)
        j, k = torch.empty_like(d), torch.empty_like(d)
        torch.cuda.synchronize()
        ctx.graph_capture(d.data_ptr(), j.data_ptr(), k.data_ptr(), mixed=case["mixed"] > 0.0)
        return {"call": call, "handle": ctx, "stream": torch.cuda.ExternalStream(ctx.stream()), "d": d, "j": j, "k": k}
    d = _density(ctx.M, seed).cpu().numpy()
    if call == "incremental":
        inc = E.Incremental(ctx, opts, exact_rebuild_interval=1000, delta_density_threshold=case["den"])
        inc.update(d)
        step = _density(ctx.M, seed + 1, scale=1e-3).cpu().numpy()
        return {"call": call, "inc": inc, "d": [d + step, d], "at": 0}
    return {"call": call, "plan": E.DirectPlan(ctx, ctx.profile()), "opts": opts, "d": d}


def run(state):
    call = state["call"]
    if call == "graph":
        cur = torch.cuda.current_stream()
        state["stream"].wait_stream(cur)
        state["handle"].graph_launch()
        cur.wait_stream(state["stream"])
        return {"J": state["j"], "K": state["k"]}
    if call == "onee":
        m = E.evaluate_one_electron_matrices_sph_into(state["mol"], state["plan"])
        return {"S": m.overlap, "T": m.kinetic, "V": m.nuclear}
    if call == "incremental":
        # an SCF step: the next density in, the updated G back
        state["inc"].update(state["d"][state["at"]])
        state["at"] ^= 1
        return {"G": state["inc"].g()}
    if call == "g":
        return {"G": E.build_rhf_g(state["plan"], state["d"], state["opts"]).g}
    if call == "j":
        return {"J": E.build_coulomb_j(state["plan"], state["d"], state["opts"]).j}
    return state["plan"].context.jk(state["d"], want=("J", "K"), options=state["opts"])


def work(case):
    """Matrices in and out once; flops of the algorithm's operation count for
    the surviving quartets (two-electron) or per primitive pair and nucleus."""
    mols, call = _molecules(case), case["call"]
    n2 = sum(m.n_sph ** 2 for m in mols)
    if call == "onee":
        mol = mols[0]
        prims = sum(len(s.exponents) * (s.L + 1) * (s.L + 2) // 2 for s in mol.shells)
        return {"bytes": 24.0 * n2, "flops": prims * prims / 2.0 * (60.0 + 20.0 * len(mol.charges))}
    flops = 0.0
    for m in mols:
        ctx = E.Context(m).plan(_options(case))
        flops += ctx.profile()["flops"]
        ctx.close()
    arrays = {"g": 2, "j": 2, "jk": 3, "graph": 3, "incremental": 3}[call]
    return {"bytes": 8.0 * arrays * n2, "flops": flops}


# ---------------------------------------------------------------------------
# Values in 64 bits by another method: McMurchie-Davidson Hermite expansions
# over all primitive pairs, unscreened, in torch.

def _moved(mol, shift):
    xyz = mol.coords + shift
    out = MOL.Molecule(mol.name, mol.charges, xyz)
    out.shells = [MOL.ShellSpec(tuple(float(v) for v in xyz[s.atom]), s.L, s.exponents, s.coefficients, s.atom)
                  for s in mol.shells]
    return out


def _carts(L):
    return [(x, y, L - x - y) for x in range(L, -1, -1) for y in range(L - x, -1, -1)]


def _odd(n):
    return math.prod(range(n, 0, -2)) if n > 0 else 1


def _solid(L):
    """Rows m = -L..L (x, y, z for p) of the real solid harmonics over the
    Cartesian monomials, each row r^L-normalised by its Gaussian self-overlap
    in units where x^L y^M z^N with even powers counts (L-1)!!(M-1)!!(N-1)!!."""
    s3, s5, s15 = math.sqrt(3.0), math.sqrt(5.0), math.sqrt(15.0)
    rows = {
        0: [{(0, 0, 0): 1}],
        1: [{(1, 0, 0): 1}, {(0, 1, 0): 1}, {(0, 0, 1): 1}],
        2: [{(1, 1, 0): 1}, {(0, 1, 1): 1}, {(0, 0, 2): 2, (2, 0, 0): -1, (0, 2, 0): -1}, {(1, 0, 1): 1},
            {(2, 0, 0): 1, (0, 2, 0): -1}],
        3: [{(2, 1, 0): 3, (0, 3, 0): -1}, {(1, 1, 1): s15}, {(0, 1, 2): 4, (2, 1, 0): -1, (0, 3, 0): -1},
            {(0, 0, 3): 2, (2, 0, 1): -3, (0, 2, 1): -3}, {(1, 0, 2): 4, (3, 0, 0): -1, (1, 2, 0): -1},
            {(2, 0, 1): s5, (0, 2, 1): -s5}, {(3, 0, 0): s3, (1, 2, 0): -3 * s3}],
    }[L]
    carts = _carts(L)
    out = np.zeros((2 * L + 1, len(carts)))
    for i, r in enumerate(rows):
        for c, v in r.items():
            out[i, carts.index(c)] = v
    gram = np.array([[math.prod(_odd(p + q - 1) if (p + q) % 2 == 0 else 0 for p, q in zip(a, b)) for b in carts]
                     for a in carts], dtype=float)
    return out / np.sqrt(np.einsum("ic,cd,id->i", out, gram, out))[:, None]


def _radial(shell):
    """Primitive coefficients of a unit-norm contracted shell."""
    a, c, L = shell.exponents, shell.coefficients, shell.L
    k = c * a ** (0.5 * L + 0.75)
    p = a[:, None] + a[None, :]
    return k / math.sqrt(np.einsum("i,j,ij->", k, k, (math.pi / p) ** 1.5 / (2.0 * p) ** L))


def _herms(L):
    return [(t, u, v) for t in range(L + 1) for u in range(L + 1 - t) for v in range(L + 1 - t - u)]


def _expansion(a, b, ra, rb, la, lb):
    """E[axis][i][j][t] of primitive pairs (vectors a, b; centres N x 3)."""
    p, ab = a + b, ra - rb
    P = (a[:, None] * ra + b[:, None] * rb) / p[:, None]
    out = []
    for x in range(3):
        pa, pb, h = P[:, x] - ra[:, x], P[:, x] - rb[:, x], 0.5 / p
        e = {(0, 0): [torch.exp(-a * b / p * ab[:, x] ** 2)]}

        def step(src, d):
            n = len(src)
            get = lambda t: src[t] if 0 <= t < n else torch.zeros_like(d)  # noqa: E731
            return [h * get(t - 1) + d * get(t) + (t + 1) * get(t + 1) for t in range(n + 1)]

        for i in range(la):
            e[i + 1, 0] = step(e[i, 0], pa)
        for i in range(la + 1):
            for j in range(lb):
                e[i, j + 1] = step(e[i, j], pb)
        out.append(e)
    return p, P, out


def _pair_classes(mol, dev):
    """Per class (la, lb): primitive pairs of all shell pairs i >= j with the
    Hermite expansions of their spherical products."""
    t = lambda v: torch.as_tensor(np.asarray(v), device=dev)  # noqa: E731
    sh = mol.shells
    off = np.concatenate([[0], np.cumsum([2 * s.L + 1 for s in sh])])
    rad = [_radial(s) for s in sh]
    classes = {}
    for la in sorted({s.L for s in sh}):
        for lb in sorted({s.L for s in sh}):
            pairs = [(i, j) for i in range(len(sh)) for j in range(i + 1) if sh[i].L == la and sh[j].L == lb]
            if not pairs:
                continue
            ex = [[], [], [], [], [], []]
            for k, (i, j) in enumerate(pairs):
                na, nb = len(rad[i]), len(rad[j])
                for lst, v in zip(ex, (np.repeat(sh[i].exponents, nb), np.tile(sh[j].exponents, na),
                                       np.repeat(rad[i], nb) * np.tile(rad[j], na), np.full(na * nb, k),
                                       np.tile(sh[i].center, (na * nb, 1)), np.tile(sh[j].center, (na * nb, 1)))):
                    lst.append(v)
            a, b, w, seg, ra, rb = (t(np.concatenate(v)) for v in ex)
            p, P, e = _expansion(a, b, ra, rb, la, lb)
            cart = torch.stack([torch.stack([torch.stack(
                [_term(e, ca, cb, h, p) for h in _herms(la + lb)], 1) for cb in _carts(lb)], 1) for ca in _carts(la)], 1)
            sph = torch.einsum("sa,tb,nabh->nsth", t(_solid(la)), t(_solid(lb)), cart) * w[:, None, None, None]
            rows = np.array([[(off[i] + s, off[j] + u) for s in range(2 * la + 1) for u in range(2 * lb + 1)]
                             for i, j in pairs])
            classes[la, lb] = {"L": la + lb, "p": p, "P": P, "seg": seg, "n": len(pairs), "E": sph.flatten(1, 2),
                               "ao": t(rows.reshape(-1, 2)), "a": a, "b": b, "ra": ra, "rb": rb, "w": w,
                               "same": t(np.array([1.0 if i == j else 2.0 for i, j in pairs]).repeat(rows.shape[1]))}
    return classes


def _term(e, ca, cb, h, like):
    v = None
    for x in range(3):
        row = e[x][ca[x], cb[x]]
        if h[x] >= len(row):
            return torch.zeros_like(like)
        v = row[h[x]] if v is None else v * row[h[x]]
    return v


def _boys(L, T):
    """F_0..F_L: ascending series and downward recursion below 35, erf and
    upward recursion above."""
    lo = T.clamp(max=35.0)
    ex = torch.exp(-lo)
    term = torch.full_like(lo, 1.0 / (2 * L + 1))
    acc = term.clone()
    steps = int(60 + 3 * float(lo.max())) if T.numel() else 0
    for i in range(1, steps):
        term = term * (2.0 * lo / (2 * L + 2 * i + 1))
        acc += term
    down = [ex * acc]
    for n in range(L, 0, -1):
        down.append((2.0 * lo * down[-1] + ex) / (2 * n - 1))
    down.reverse()
    hi = T.clamp(min=35.0)
    exh, up = torch.exp(-hi), [0.5 * torch.sqrt(math.pi / hi) * torch.erf(torch.sqrt(hi))]
    for n in range(L):
        up.append(((2 * n + 1) * up[-1] - exh) / (2.0 * hi))
    return [torch.where(T < 35.0, d, u) for d, u in zip(down, up)]


def _hermite(L, alpha, R):
    """R_tuv (t+u+v <= L) of exponent alpha and vectors R (... x 3)."""
    f = _boys(L, alpha * (R * R).sum(-1))
    cur = {}
    for n in range(L, -1, -1):
        new = {(0, 0, 0): (-2.0 * alpha) ** n * f[n]}
        for h in _herms(L - n):
            if h == (0, 0, 0):
                continue
            x = next(k for k in range(3) if h[k])
            one = tuple(v - (k == x) for k, v in enumerate(h))
            v = R[..., x] * cur[one]
            if one[x]:
                two = tuple(v2 - (k == x) for k, v2 in enumerate(one))
                v = v + one[x] * cur[two]
            new[h] = v
        cur = new
    return cur


def _eri_rows(bra, ket):
    """(rows of bra) x (rows of ket) matrix of (ab|cd)."""
    hb, hk, L = _herms(bra["L"]), _herms(ket["L"]), bra["L"] + ket["L"]
    nab, ncd, nk = bra["E"].shape[1], ket["E"].shape[1], len(ket["p"])
    out = torch.zeros(bra["n"], nab, ket["n"] * ncd, dtype=F64, device=bra["p"].device)
    sign = torch.tensor([(-1.0) ** sum(h) for h in hk], dtype=F64, device=bra["p"].device)
    ek = (ket["E"] * sign).transpose(1, 2)
    step = max(1, int(4e6 / (len(hb) * len(hk) * nk) * 8))
    for b0 in range(0, len(bra["p"]), step):
        sl = slice(b0, b0 + step)
        p, q = bra["p"][sl, None], ket["p"][None, :]
        r = _hermite(L, p * q / (p + q), bra["P"][sl, None, :] - ket["P"][None, :, :])
        pre = 2.0 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q))
        m = torch.stack([torch.stack([r[tuple(x + y for x, y in zip(h, g))] for g in hk], -1) for h in hb], -2)
        nb = m.shape[0]
        m = (m * pre[..., None, None]).transpose(0, 1).reshape(nk, nb * len(hb), len(hk)) @ ek
        c = torch.zeros(ket["n"], nb * len(hb), ncd, dtype=F64, device=m.device).index_add_(0, ket["seg"], m)
        c = c.reshape(ket["n"], nb, len(hb), ncd).permute(1, 2, 0, 3).reshape(nb, len(hb), -1)
        out.index_add_(0, bra["seg"][sl], bra["E"][sl] @ c)
    return out.reshape(bra["n"] * nab, ket["n"] * ncd)


def _exact_jk(mol, D):
    dev = D.device
    cl = list(_pair_classes(mol, dev).values())
    n = mol.n_sph
    ao = torch.cat([c["ao"] for c in cl])
    start = np.concatenate([[0], np.cumsum([len(c["ao"]) for c in cl])])
    P = torch.empty(len(ao), len(ao), dtype=F64, device=dev)
    for x in range(len(cl)):
        for y in range(x + 1):
            v = _eri_rows(cl[x], cl[y])
            P[start[x]:start[x + 1], start[y]:start[y + 1]] = v
            P[start[y]:start[y + 1], start[x]:start[x + 1]] = v.T
    row = torch.empty(n, n, dtype=torch.long, device=dev)
    r = torch.arange(len(ao), device=dev)
    row[ao[:, 0], ao[:, 1]] = r
    row[ao[:, 1], ao[:, 0]] = r
    # every AO pair (k, l), k and l free, reads its row of P
    J = (P[:, :] @ (torch.cat([c["same"] for c in cl]) * D[ao[:, 0], ao[:, 1]]))[row]
    K = torch.stack([torch.einsum("jkl,jl->k", P[row[i]][:, row.reshape(-1)].reshape(n, n, n), D) for i in range(n)])
    return J, K


def _exact_onee(mol, dev):
    n = mol.n_sph
    S, T, V = (torch.zeros(n, n, dtype=F64, device=dev) for _ in range(3))
    nuc = torch.as_tensor(mol.coords, device=dev, dtype=F64)
    Z = torch.as_tensor(np.asarray(mol.charges, dtype=float), device=dev)
    for (la, lb), c in _pair_classes(mol, dev).items():
        p, b, L = c["p"], c["b"], c["L"]
        herms = _herms(L)
        v = torch.zeros(len(p), len(herms), dtype=F64, device=dev)
        step = max(1, int(4e7 / (len(herms) * len(Z))))
        for k in range(0, len(p), step):
            sl = slice(k, k + step)
            r = _hermite(L, p[sl, None].expand(-1, len(Z)), c["P"][sl, None, :] - nuc[None])
            v[sl] = torch.stack([(r[h] * Z).sum(1) for h in herms], 1)
        _, _, e = _expansion(c["a"], b, c["ra"], c["rb"], la, lb + 2)
        s1 = [{ij: row[0] for ij, row in ex.items()} for ex in e]

        def kin(x, i, j):
            out = b * (2 * j + 1) * s1[x][i, j] - 2.0 * b * b * s1[x][i, j + 2]
            return out - 0.5 * j * (j - 1) * s1[x][i, j - 2] if j > 1 else out

        s, t = [], []
        for ca in _carts(la):
            for cb in _carts(lb):
                o = [s1[x][ca[x], cb[x]] for x in range(3)]
                k = [kin(x, ca[x], cb[x]) for x in range(3)]
                s.append(o[0] * o[1] * o[2])
                t.append(k[0] * o[1] * o[2] + o[0] * k[1] * o[2] + o[0] * o[1] * k[2])
        sa, sb = (torch.as_tensor(_solid(l), device=dev) for l in (la, lb))
        pre = c["w"] * (math.pi / p) ** 1.5
        shape = (len(p), len(_carts(la)), len(_carts(lb)))
        for X, val in ((S, s), (T, t)):
            val = torch.einsum("sa,tb,nab->nst", sa, sb, torch.stack(val, 1).reshape(shape)) * pre[:, None, None]
            _scatter(X, c, val.flatten(1))
        _scatter(V, c, -(2.0 * math.pi / p)[:, None] * torch.einsum("nch,nh->nc", c["E"], v))
    return S, T, V


def _scatter(X, c, val):
    rows = torch.zeros(c["n"], val.shape[1], dtype=F64, device=val.device).index_add_(0, c["seg"], val).reshape(-1)
    X[c["ao"][:, 0], c["ao"][:, 1]] = rows
    X[c["ao"][:, 1], c["ao"][:, 0]] = rows


def exact(case, seed):
    """None where the four-index values would not fit or take too long."""
    mols, call = _molecules(case), case["call"]
    dev = torch.device("cuda")
    if call == "onee":
        mol = mols[0]
        shift = np.random.default_rng(seed).normal(scale=0.02, size=mol.coords.shape)
        S, T, V = _exact_onee(_moved(mol, shift), dev)
        return {"S": S, "T": T, "V": V}
    if sum(m.n_sph ** 4 for m in mols) > 250 ** 4 or max(s.L for m in mols for s in m.shells) > 2:
        return None
    if case["mol"] == "batch":
        js, ks = zip(*(_exact_jk(m, _density(m.n_sph, seed + 7919 * k)) for k, m in enumerate(mols)))
        return {"J": torch.cat([j.reshape(-1) for j in js]), "K": torch.cat([k.reshape(-1) for k in ks])}
    D = _density(mols[0].n_sph, seed)
    if call == "incremental":
        D = D + _density(mols[0].n_sph, seed + 1, scale=1e-3)
    J, K = _exact_jk(mols[0], D)
    return {"J": J, "K": K} if call in ("graph", "jk") else {"J": J} if call == "j" else {"G": J - 0.5 * K}
