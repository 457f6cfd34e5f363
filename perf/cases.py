"""The measured workloads of the two-electron path, each one call a user's
program makes: direct J/K builds (host arrays or device tensors, FP64 or
FP32-mixed, symmetric or not), density-direct gradients, the dense, packed
and row-built tensors, density fitting and molecule batches.

Molecules are synthetic, as in the repository's own benchmarks: atoms placed
uniformly at random in a cube with a smallest separation, every atom with the
same shells, even-tempered exponents and random contraction coefficients, and
densities D = C C^T.  ``exact`` evaluates the same quantities with a plain
McMurchie-Davidson scheme in 64 bits in torch.
"""
import functools
import itertools
import math

import numpy as np
import torch

import integral_b200 as ib

L_OF = {"s": 0, "p": 1, "d": 2, "f": 3, "g": 4}

# Bases of the repository's configurations: letters, primitives per shell,
# smallest exponent, ratio, smallest coefficient, cubic bohr per atom,
# smallest separation.
BASES = {
    "spd": ("sssppd", 3, 0.10, 2.5, 0.2, 125.0, 1.8),  # the J/K benchmark
    "sp": ("ssspp", 3, 0.15, 3.0, 0.2, 85.0, 1.5),  # the dense tensor
    "grad": ("ssppd", 3, 0.12, 2.5, 0.2, 138.0, 1.8),  # the gradient
    "spdf": ("sssppddf", 4, 0.08, 2.2, 0.1, 164.0, 1.8),  # the spherical f recipe
    "f": ("ssppdf", 3, 0.12, 2.5, 0.2, 68.0, 1.5),  # density fitting, f gradients
    "g": ("ssppdfg", 3, 0.10, 2.4, 0.2, 15.6, 1.6),  # the compact batch molecules
}
AUX = "spdfspd"  # single primitives 0.2 * 1.8^k, the density-fitting basis

DEFAULTS = dict(op="jk", basis="spd", atoms=4, kinds="cartesian", dens=1, symmetric=True, exchange=True, tau=1e-12,
                mixed=False, omega=0.0, share=1, molecules=1)


def _case(name=None, **kw):
    c = dict(DEFAULTS, **kw)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # one small molecule through the host-array call: launches and latency
        _case("jk_host_small", op="jk_host", atoms=3),
        # SCF iteration of a mid-size molecule in double precision
        _case("jk_fp64", atoms=16),
        # the headline call: four densities, mixed precision, a larger molecule
        _case("jk_mixed", atoms=32, dens=4, mixed=True),
        # spherical basis with f shells, two densities, mixed precision
        _case("jk_spdf_mixed", basis="spdf", kinds="spherical", atoms=8, dens=2, tau=1e-11, mixed=True),
        # transition densities (not symmetric), as response solvers pass them
        _case("jk_nonsymmetric", atoms=11, dens=2, symmetric=False),
        # g shells in a compact molecule
        _case("jk_g", basis="g", kinds="spherical", atoms=5, tau=1e-11),
        # nuclear gradient in double precision, odd atom count
        _case("grad_fp64", op="grad", basis="grad", atoms=11),
        # nuclear gradient of a larger molecule, mixed precision
        _case("grad_mixed", op="grad", basis="grad", atoms=18, mixed=True),
        # gradient over spherical f shells
        _case("grad_f_spherical", op="grad", basis="f", kinds="spherical", atoms=5, tau=1e-11),
        # the whole tensor of a small molecule, as a correlated method stores it
        _case("eri_dense", op="eri", basis="sp", atoms=6),
        # density fitting: three-centre tensor and metric
        _case("df_build", op="df", basis="f", kinds="spherical", atoms=8),
        # many small molecules in one call, J/K and gradients
        _case("batch_jk_grad", op="batch", basis="f", kinds="spherical", atoms=5, molecules=8, tau=1e-11, mixed=True),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo - 0.49), math.log(hi + 0.49)))))))


def draw(rng):
    """A case of the same ranges: an operation, then its basis, size and options."""
    op = rng.choice(["jk", "jk", "jk", "jk_host", "grad", "grad", "eri", "packed", "rows", "df", "batch"])
    c = dict(op=op, tau=rng.choice([1e-10, 1e-11, 1e-12]))
    if op in ("jk", "jk_host"):
        c["basis"] = rng.choice(["spd", "spd", "spd", "grad", "spdf", "f", "g"])
        c["kinds"] = rng.choice(["cartesian", "cartesian", "spherical"])
        c["dens"] = rng.choice([1, 1, 2, 3, 4, 5])
        c["symmetric"] = rng.random() < 0.8
        c["exchange"] = rng.random() < 0.85
        c["mixed"] = rng.random() < 0.5
        top = {"spd": 28, "grad": 28, "spdf": 6, "f": 8, "g": 4}[c["basis"]]
        if not c["mixed"] and top > 20:
            top = 20
        if c["kinds"] != "spherical" and c["basis"] in ("spdf", "f", "g"):
            c["kinds"] = rng.choice(["spherical", "spherical", "cartesian"])
            top = top if c["kinds"] == "spherical" else {"spdf": 4, "f": 5, "g": 2}[c["basis"]]
        if not c["symmetric"] and top > 10:
            top = 10
        if rng.random() < 0.1:
            c["kinds"], top = "mixed", min(top, 6)
        c["atoms"] = _log_int(rng, 2, top)
        c["share"] = rng.choice([1, 1, 1, 1, 2, 4]) if op == "jk" else 1
    elif op == "grad":
        c["basis"] = rng.choice(["grad", "grad", "spd", "f"])
        c["kinds"] = rng.choice(["cartesian", "cartesian", "spherical"])
        c["mixed"] = rng.random() < 0.5
        c["omega"] = rng.choice([0.0, 0.0, 0.0, 0.3])
        top = {"grad": 14, "spd": 12, "f": 4}[c["basis"]]
        if c["kinds"] == "spherical" and c["basis"] != "f":
            top = 9
        c["atoms"] = _log_int(rng, 2, top)
    elif op in ("eri", "packed", "rows"):
        c["basis"] = rng.choice(["sp", "sp", "grad", "f"])
        c["kinds"] = rng.choice(["cartesian", "spherical"])
        c["omega"] = rng.choice([0.0, 0.0, 0.3]) if op != "packed" else 0.0
        c["atoms"] = _log_int(rng, 2, {"sp": 6, "grad": 3, "f": 2}[c["basis"]])
    elif op == "df":
        c["basis"] = rng.choice(["f", "f", "spd"])
        c["kinds"] = rng.choice(["spherical", "spherical", "cartesian"])
        c["atoms"] = _log_int(rng, 2, 8 if c["kinds"] == "spherical" else 6)
    else:
        c["basis"] = rng.choice(["grad", "f"])
        c["kinds"] = "spherical"
        c["atoms"] = rng.randint(2, 5)
        c["molecules"] = _log_int(rng, 2, 8)
        c["mixed"] = rng.random() < 0.5
    return _case(**c)


# ------------------------------------------------------------------- inputs

def _n_func(l, spherical):
    return 2 * l + 1 if spherical else (l + 1) * (l + 2) // 2


def _place(rng, atoms, side, sep):
    pts = []
    while len(pts) < atoms:
        p = rng.uniform(0.0, side, size=3)
        if all(np.sum((p - q) ** 2) >= sep * sep for q in pts):
            pts.append(p)
    return pts


def _molecule(rng, case, atoms):
    letters, nprim, base, ratio, lo, volume, sep = BASES[case["basis"]]
    shells = []
    for c in _place(rng, atoms, (volume * atoms) ** (1.0 / 3.0), sep):
        for x in letters:
            # "mixed": Cartesian d shells, all others spherical
            sph = case["kinds"] == "spherical" or (case["kinds"] == "mixed" and x != "d")
            shells.append(dict(l=L_OF[x], spherical=sph, center=[float(v) for v in c],
                               exps=[base * ratio ** k for k in range(nprim)],
                               coefs=[float(v) for v in rng.uniform(lo, 1.0, size=nprim)]))
    return shells


def _aux(rng, case, shells):
    centers = list(dict.fromkeys(tuple(s["center"]) for s in shells))
    return [dict(l=L_OF[x], spherical=case["kinds"] != "cartesian", center=list(c),
                 exps=[0.2 * 1.8 ** k * float(rng.uniform(0.8, 1.2))], coefs=[1.0])
            for c in centers for k, x in enumerate(AUX)]


def _nao(shells):
    return sum(_n_func(s["l"], s["spherical"]) for s in shells)


def _densities(rng, nao, count, symmetric):
    out = []
    occ = max(1, nao // 4)
    for _ in range(count):
        C = rng.normal(0.0, 1.0 / math.sqrt(nao), size=(nao, occ))
        if symmetric:
            D = C @ C.T
            D = 0.5 * (D + D.T)
        else:
            D = C @ rng.normal(0.0, 1.0 / math.sqrt(nao), size=(nao, occ)).T
        out.append(D)
    return np.ascontiguousarray(out)


def _inputs(case, seed):
    """Molecules, densities and the auxiliary basis, from the seed alone."""
    rng = np.random.default_rng(seed)
    if case["op"] == "batch":
        # uneven molecules: 2 .. atoms atoms each, at least one of the largest
        sizes = [case["atoms"] - (m % max(1, case["atoms"] - 1)) for m in range(case["molecules"])]
        mols = [_molecule(rng, case, n) for n in sizes]
        return dict(molecules=mols, dens=[_densities(rng, _nao(m), 1, True)[0] for m in mols])
    shells = _molecule(rng, case, case["atoms"])
    got = dict(shells=shells)
    if case["op"] in ("jk", "jk_host"):
        got["dens"] = _densities(rng, _nao(shells), case["dens"], case["symmetric"])
    elif case["op"] == "grad":
        got["dens"] = _densities(rng, _nao(shells), 1, True)[0]
    elif case["op"] == "df":
        got["aux"] = _aux(rng, case, shells)
    return got


def prepare(case, seed):
    inp = _inputs(case, seed)
    s = dict(case=case)
    op = case["op"]
    if op == "batch":
        s["batch"] = ib.MoleculeBatch(inp["molecules"])
        s["dens"] = inp["dens"]
        return s
    basis = ib.Basis(inp["shells"])
    basis.plan()
    s["basis"] = basis
    if op in ("jk", "jk_host"):
        s["dc"] = basis.direct_contractor()
        s["dens"] = inp["dens"]
        if op == "jk":
            s["stream"] = torch.cuda.Stream()
            s["D"] = torch.from_numpy(inp["dens"]).cuda()
            s["J"] = torch.empty_like(s["D"])
            s["K"] = torch.empty_like(s["D"]) if case["exchange"] else None
            nsh = len(inp["shells"])
            s["bras"] = None if case["share"] == 1 else np.arange(0, nsh * (nsh + 1) // 2, case["share"], dtype=np.uint32)
            torch.cuda.synchronize()
    elif op == "grad":
        s["gc"] = basis.direct_grad_contractor()
        D = inp["dens"]
        s["density"] = s["gc"].density([ib.GradDensityTerm(0.5, D, D)], [ib.GradDensityTerm(-0.25, D, D)])
        s["kernel"] = ib.EriKernel.Erf(case["omega"]) if case["omega"] else None
    elif op == "rows":
        s["builder"] = basis.eri_builder()
        if case["omega"]:
            s["builder"].kernel(ib.EriKernel.Erf(case["omega"]))
    elif op == "packed":
        s["builder"] = basis.packed_eri_builder()
    elif op == "df":
        s["aux"] = ib.Basis(inp["aux"])
        s["builder"] = basis.eri_3c_builder(s["aux"])
    return s


def run(state):
    case = state["case"]
    op = case["op"]
    prec = 1 if case["mixed"] else 0
    if op == "jk":
        st = state["stream"]
        with torch.cuda.stream(st):
            state["J"].zero_()
            if case["exchange"]:
                state["K"].zero_()
            state["dc"].jk_device(state["D"].data_ptr(), case["dens"], state["J"].data_ptr(),
                                  state["K"].data_ptr() if case["exchange"] else 0, case["tau"],
                                  want_exchange=case["exchange"], precision=prec, bras=state["bras"],
                                  stream=st.cuda_stream)
        return {"J": state["J"], "K": state["K"]}
    if op == "jk_host":
        J, K = state["dc"].jk(state["dens"], case["tau"], want_exchange=case["exchange"], precision=prec)
        return {"J": J, "K": K}
    if op == "grad":
        return {"grad": state["gc"].contract(state["density"], kernel=state["kernel"], threshold=case["tau"],
                                             precision=prec)}
    if op == "eri":
        b = state["basis"]
        return {"eri": b.eri_kernel(ib.EriKernel.Erf(case["omega"])) if case["omega"] else b.eri()}
    if op == "rows":
        return {"eri": state["builder"].build()}
    if op == "packed":
        return {"eri": state["builder"].build(case["tau"])}
    if op == "df":
        return {"eri_3c": state["builder"].build(), "eri_2c": state["aux"].eri_2c()}
    J, K, G = state["batch"].jk_grad(state["dens"], case["tau"], precision=prec)
    return {"J": np.concatenate([m.reshape(-1) for m in J]), "K": np.concatenate([m.reshape(-1) for m in K]),
            "grad": np.concatenate(G)}


# --------------------------------------------------------------------- work

def _prim_flops(la, lb, lc, ld):
    """One primitive quartet: its header, the roots and weights, the per-axis
    vertical recurrences and the sum into the [e0|f0] table, whose elements of
    one (ex, ey, fx, fy) share a product."""
    ne, nf = la + lb, lc + ld
    n = (ne + nf) // 2 + 1
    rng = lambda lo, hi: sum((d + 1) * (d + 2) // 2 for d in range(lo, hi + 1))  # noqa: E731
    return 40 + 2 * n * 34 + n * (12 + 3 * 4 * (ne + 1) * (nf + 1) + 3 * rng(la, ne) * rng(lc, nf))


def _pair_estimates(shells):
    """Per canonical shell pair: class, primitive pairs, and an estimate of
    its Schwarz bound (the s-type self-repulsion of its largest primitive
    pair), for counting the quartets that pass the screen."""
    by = {}
    for i in range(len(shells)):
        for j in range(i + 1):
            a, b = (shells[i], shells[j]) if shells[i]["l"] >= shells[j]["l"] else (shells[j], shells[i])
            d2 = sum((x - y) ** 2 for x, y in zip(a["center"], b["center"]))
            ea, eb = np.array(a["exps"])[:, None], np.array(b["exps"])[None, :]
            p = ea + eb
            ca = np.array(a["coefs"])[:, None] * (2 * ea / math.pi) ** 0.75
            cb = np.array(b["coefs"])[None, :] * (2 * eb / math.pi) ** 0.75
            q = np.abs(ca * cb) * np.exp(-ea * eb / p * d2) * np.sqrt(34.9868 / (p * p * np.sqrt(2 * p)))
            by.setdefault((a["l"], b["l"]), []).append((float(q.max()), p.size))
    return by


@functools.lru_cache(maxsize=None)
def _quartet_flops(key):
    """Flops of the quartets of one molecule of typical geometry that pass the
    screen: primitive work (weight `grad`: the three raised classes in its
    place) and 24 flops per block element and density for the J/K sums."""
    case = dict(key)
    shells = _molecule(np.random.default_rng(1234), case, case["atoms"])
    by = _pair_estimates(shells)
    tau = case["tau"] if case["op"] in ("jk", "jk_host", "grad", "batch", "packed") else 0.0
    sph = case["kinds"] != "cartesian"
    jk, grad = 0.0, 0.0
    classes = sorted(by, key=lambda c: c[0] * (c[0] + 1) // 2 + c[1])
    for x, y in itertools.combinations_with_replacement(range(len(classes)), 2):
        (lc, ld), (la, lb) = classes[x], classes[y]
        qa, qb = np.array([v[0] for v in by[(la, lb)]]), np.sort([v[0] for v in by[(lc, ld)]])
        npp = by[(la, lb)][0][1] * by[(lc, ld)][0][1]
        n = float(np.sum(len(qb) - np.searchsorted(qb, tau / qa))) if tau > 0 else float(len(qa) * len(qb))
        n *= 0.5 if x == y else 1.0
        block = np.prod([float(_n_func(l, sph)) for l in (la, lb, lc, ld)])
        jk += n * (npp * _prim_flops(la, lb, lc, ld) + 24.0 * block * case["dens"])
        grad += n * (npp * (_prim_flops(la + 1, lb, lc, ld) + _prim_flops(la, lb, lc + 1, ld)) + 36.0 * block)
    return float(jk), float(grad)


def _basis_key(case, **kw):
    c = {k: v for k, v in case.items() if k != "name"}
    c.update(kw)
    return tuple(sorted(c.items()))


def work(case):
    op = case["op"]
    if op == "batch":
        inp = _inputs(case, 1234)
        flops = sum(sum(_quartet_flops(_basis_key(case, atoms=len({tuple(s["center"]) for s in m}))))
                    for m in inp["molecules"])
        return {"bytes": 8.0 * sum(4 * _nao(m) ** 2 for m in inp["molecules"]), "flops": flops}
    inp = _inputs(case, 1234)
    n = _nao(inp["shells"])
    if op == "df":
        na = _nao(inp["aux"])
        flops = 0.0
        for (la, lb), v in _pair_estimates(inp["shells"]).items():
            for s in inp["aux"]:
                flops += sum(x[1] for x in v) * _prim_flops(la, lb, s["l"], 0)
        for s, t in itertools.combinations_with_replacement(inp["aux"], 2):
            flops += _prim_flops(s["l"], 0, t["l"], 0)
        return {"bytes": 8.0 * (n * n * na + na * na), "flops": flops}
    jk, grad = _quartet_flops(_basis_key(case))
    if op == "grad":
        return {"bytes": 8.0 * n * n, "flops": grad}
    if op in ("jk", "jk_host"):
        return {"bytes": 8.0 * n * n * case["dens"] * (3 if case["exchange"] else 2), "flops": jk / case["share"]}
    m = n * (n + 1) // 2
    return {"bytes": 8.0 * (m * (m + 1) // 2 if op == "packed" else n ** 4), "flops": jk}


def tolerance(case):
    """FP64 sums agree to rounding (the screened remainder is the same list);
    a mixed call rounds its small quartets to 24 bits."""
    if case["mixed"]:
        return {"rel": 1e-6, "max": 1e-5}
    if case["basis"] in ("f", "g", "spdf") or case["op"] == "df":
        return {"rel": 1e-10, "max": 1e-8}
    return {"rel": 1e-11, "max": 1e-9}


# -------------------------------------------------------------------- exact
#
# McMurchie-Davidson: shell pairs expand in Hermite Gaussians, (ab|cd) =
# E_ab R E_cd^T with R the Hermite Coulomb integrals, per primitive quartet.

def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _cart(l):
    return [(x, y, l - x - y) for x in range(l, -1, -1) for y in range(l - x, -1, -1)]


def _dfact(n):
    return math.prod(range(n, 0, -2)) if n > 0 else 1


@functools.lru_cache(maxsize=None)
def _solid(l):
    """Real solid harmonics over the Cartesian components, rows normalised to
    one for (l,0,0)-normalised Gaussians; p rows x, y, z, others ascending m."""
    comps = _cart(l)
    rows = []
    for m in [1, -1, 0] if l == 1 else range(-l, l + 1):
        M = abs(m)
        poly = dict.fromkeys(comps, 0.0)
        for k in range((l - M) // 2 + 1):
            g = (-1.0) ** k * math.comb(l, k) * math.comb(2 * l - 2 * k, l) * math.perm(l - 2 * k, M)
            for a, b in itertools.product(range(k + 1), repeat=2):
                if a + b > k:
                    continue
                mult = math.factorial(k) / (math.factorial(a) * math.factorial(b) * math.factorial(k - a - b))
                for q in range(M + 1):
                    if (q % 2 == 1) != (m < 0):
                        continue
                    sign = -1.0 if q % 4 in (2, 3) else 1.0
                    poly[(2 * a + M - q, 2 * b + q, 2 * (k - a - b) + l - 2 * k - M)] += g * mult * math.comb(M, q) * sign
        v = np.array([poly[c] for c in comps])
        ov = np.array([[0.0 if any((x + y) % 2 for x, y in zip(c, d)) else
                        math.prod(_dfact(x + y - 1) for x, y in zip(c, d)) for d in comps] for c in comps])
        rows.append(v / math.sqrt(v @ ov @ v / _dfact(2 * l - 1)))
    return np.array(rows)


def _to_func(shell):
    n = len(_cart(shell["l"]))
    return torch.tensor(_solid(shell["l"]) if shell["spherical"] else np.eye(n), dtype=torch.float64, device=_dev())


def _herm(L):
    return [(t, u, v) for N in range(L + 1) for (t, u, v) in _cart(N)]


@functools.lru_cache(maxsize=None)
def _herm_index(L):
    return {h: k for k, h in enumerate(_herm(L))}


def _hermite_1d(a, b, ab, la, lb):
    """E[i][j][t] (tensors like a) of x_A^i x_B^j exp(-a x_A^2 - b x_B^2)."""
    p = a + b
    pa, pb = -b / p * ab, a / p * ab
    zero = torch.zeros_like(p)
    E = {(0, 0): [torch.exp(-a * b / p * ab * ab)]}
    get = lambda e, t: e[t] if 0 <= t < len(e) else zero  # noqa: E731
    for i, j in itertools.product(range(la + 1), range(lb + 1)):
        if (i, j) == (0, 0):
            continue
        src, x = (E[(i - 1, j)], pa) if i > 0 else (E[(i, j - 1)], pb)
        E[(i, j)] = [get(src, t - 1) / (2 * p) + x * get(src, t) + (t + 1) * get(src, t + 1) for t in range(i + j + 1)]
    return E


def _pair_class(shells, pairs, deriv, unit):
    """Hermite expansions of shell pairs of one class: exponents [n, k],
    centres [n, k, 3], E [n, k, functions (x 6 with `deriv`: d/dA, d/dB),
    hermites].  `unit`: the second shell is the constant one."""
    f = dict(dtype=torch.float64, device=_dev())
    sa = [shells[i] for i, _ in pairs]
    sb = [None if unit else shells[j] for _, j in pairs]
    la, lb = sa[0]["l"], 0 if unit else sb[0]["l"]

    def norm(s):
        return [c * (2 * e / math.pi) ** 0.75 * math.sqrt((4 * e) ** s["l"] / _dfact(2 * s["l"] - 1))
                for e, c in zip(s["exps"], s["coefs"])]

    ea = torch.tensor([s["exps"] for s in sa], **f)[:, :, None]
    ca = torch.tensor([norm(s) for s in sa], **f)[:, :, None]
    A = torch.tensor([s["center"] for s in sa], **f)
    if unit:
        eb, cb, B = torch.zeros_like(ea[:, :1, :1]), torch.ones_like(ea[:, :1, :1]), A
    else:
        eb = torch.tensor([s["exps"] for s in sb], **f)[:, None, :]
        cb = torch.tensor([norm(s) for s in sb], **f)[:, None, :]
        B = torch.tensor([s["center"] for s in sb], **f)
    n, ka, kb = len(pairs), ea.shape[1], eb.shape[2]
    ea, eb = ea.expand(n, ka, kb).reshape(n, -1), eb.expand(n, ka, kb).reshape(n, -1)
    c = (ca * cb).expand(n, ka, kb).reshape(n, -1)
    p = ea + eb
    P = (ea[..., None] * A[:, None] + eb[..., None] * B[:, None]) / p[..., None]
    up = 1 if deriv else 0
    E1 = [_hermite_1d(ea, eb, (A - B)[:, x, None], la + up, lb + up) for x in range(3)]
    hs = _herm(la + lb + up)

    def axis(x, i, j, t):
        if i < 0 or j < 0 or t > i + j:
            return None
        return E1[x][(i, j)][t]

    def element(ca_, cb_, h, shift):
        terms = [(None, ca_, cb_)]
        if shift is not None:
            which, x = shift
            l = (ca_ if which == 0 else cb_)[x]
            bump = lambda v, s: tuple(w + s if k == x else w for k, w in enumerate(v))  # noqa: E731
            e2 = 2 * (ea if which == 0 else eb)
            terms = [(e2, bump(ca_, 1), cb_) if which == 0 else (e2, ca_, bump(cb_, 1))]
            if l > 0:
                terms.append((-float(l), bump(ca_, -1), cb_) if which == 0 else (-float(l), ca_, bump(cb_, -1)))
        out = None
        for fac, u, v in terms:
            e = [axis(x, u[x], v[x], h[x]) for x in range(3)]
            if any(y is None for y in e):
                continue
            y = c * e[0] * e[1] * e[2]
            y = y if fac is None else y * fac
            out = y if out is None else out + y
        return torch.zeros_like(c) if out is None else out

    shifts = [None] if not deriv else [(w, x) for w in (0, 1) for x in range(3)]
    blocks = []
    for s in shifts:
        m = torch.stack([torch.stack([torch.stack([element(u, v, h, s) for h in hs], -1) for v in _cart(lb)], -2)
                         for u in _cart(la)], -3)  # [n, k, na, nb, h]
        m = torch.einsum("ax,nkxyh->nkayh", _to_func(sa[0]), m)
        if not unit:
            m = torch.einsum("by,nkayh->nkabh", _to_func(sb[0]), m)
        blocks.append(m.reshape(n, m.shape[1], -1, len(hs)))
    return dict(p=p, P=P, E=torch.cat(blocks, 2), L=la + lb + up)


def _boys(T, m_max):
    """F_0 .. F_m_max, stacked first: the ascending series of F_m_max and
    downward recursion below T = 30 + m_max, upward recursion above."""
    big = T > 30.0 + m_max
    t = torch.where(big, torch.ones_like(T), T)
    term = torch.full_like(t, 1.0 / (2 * m_max + 1))
    acc = term.clone()
    for k in range(1, 130 + 3 * m_max):
        term = term * (2 * t / (2 * m_max + 2 * k + 1))
        acc = acc + term
    e = torch.exp(-t)
    F = [None] * (m_max + 1)
    F[m_max] = acc * e
    for m in range(m_max - 1, -1, -1):
        F[m] = (2 * t * F[m + 1] + e) / (2 * m + 1)
    tb = torch.where(big, T, torch.full_like(T, 100.0))
    eb = torch.exp(-tb)
    G = [0.5 * torch.sqrt(math.pi / tb) * torch.erf(torch.sqrt(tb))]
    for m in range(m_max):
        G.append(((2 * m + 1) * G[m] - eb) / (2 * tb))
    return torch.stack([torch.where(big, g, f) for f, g in zip(F, G)])


@functools.lru_cache(maxsize=None)
def _r_steps(L):
    """Per degree: axis, source of degree N-1, factor and source of degree N-2."""
    steps = []
    for N in range(1, L + 1):
        ax, s1, fac, s2 = [], [], [], []
        i1 = {h: k for k, h in enumerate(_cart(N - 1))}
        i2 = {h: k for k, h in enumerate(_cart(N - 2))} if N > 1 else {}
        for h in _cart(N):
            x = next(k for k in range(3) if h[k] > 0)
            down = lambda v: tuple(w - 1 if k == x else w for k, w in enumerate(v))  # noqa: E731
            ax.append(x)
            s1.append(i1[down(h)])
            fac.append(float(h[x] - 1))
            s2.append(i2[down(down(h))] if h[x] > 1 else 0)
        steps.append(tuple(torch.tensor(v, device=_dev()) for v in (ax, s1, fac, s2)))
    return steps


@functools.lru_cache(maxsize=None)
def _r_table(La, Lb):
    idx = _herm_index(La + Lb)
    at = [[idx[tuple(x + y for x, y in zip(h, k))] for k in _herm(Lb)] for h in _herm(La)]
    sign = [(-1.0) ** sum(k) for k in _herm(Lb)]
    return torch.tensor(at, device=_dev()), torch.tensor(sign, dtype=torch.float64, device=_dev())


def _hermite_coulomb(p, q, PQ, La, Lb, omega):
    """R[batch, herm(La), herm(Lb)] with the prefactor and the ket's signs."""
    L = La + Lb
    rho = p * q / (p + q)
    pre = 2 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q))
    if omega:
        s = omega * omega / (rho + omega * omega)
        rho, pre = rho * s, pre * torch.sqrt(s)
    F = _boys(rho * (PQ * PQ).sum(-1), L)
    base = torch.stack([F[m] * pre * (-2 * rho) ** m for m in range(L + 1)])  # [m, batch]
    X = PQ.T
    lev = [base[:, None, :]]  # degree N: [m <= L - N, comps, batch]
    for N, (ax, s1, fac, s2) in enumerate(_r_steps(L), 1):
        v = X[ax][None] * lev[N - 1][1:, s1]
        if N > 1:
            v = v + fac[None, :, None] * lev[N - 2][1:L - N + 2, s2]
        lev.append(v)
    R = torch.cat([v[0] for v in lev], 0)  # [herm(L), batch]
    at, sign = _r_table(La, Lb)
    return R[at].permute(2, 0, 1) * sign


def _blocks(bra, ket, omega):
    """V[bra pairs, bra functions, ket pairs, ket functions] of two classes."""
    nb, kb = bra["p"].shape
    nk, kk = ket["p"].shape
    hb, hk = bra["E"].shape[-1], ket["E"].shape[-1]
    out = []
    step = max(1, int(3e7 // (kb * nk * kk * hb * hk)))
    kstep = max(1, min(nk, int(3e7 // (kb * kk * hb * hk))))
    for b0 in range(0, nb, step):
        b = slice(b0, min(nb, b0 + step))
        n = b.stop - b0
        row = []
        for k0 in range(0, nk, kstep):
            k = slice(k0, min(nk, k0 + kstep))
            m = k.stop - k0
            shape = (n, kb, m, kk)
            p = bra["p"][b][:, :, None, None].expand(shape).reshape(-1)
            q = ket["p"][k][None, None].expand(shape).reshape(-1)
            PQ = (bra["P"][b][:, :, None, None] - ket["P"][k][None, None]).expand(*shape, 3).reshape(-1, 3)
            R = _hermite_coulomb(p, q, PQ, bra["L"], ket["L"], omega).reshape(*shape, hb, hk)
            X = torch.einsum("nkmjxy,mjcy->nkmxc", R, ket["E"][k])
            row.append(torch.einsum("nkax,nkmxc->namc", bra["E"][b], X))
        out.append(torch.cat(row, 2))
    return torch.cat(out, 0)


def _classes(shells):
    """Canonical pairs by class of (angular momenta, kinds), each with the
    higher l first, and their AO index arrays."""
    off = np.cumsum([0] + [_n_func(s["l"], s["spherical"]) for s in shells])
    by = {}
    for i in range(len(shells)):
        for j in range(i + 1):
            a, b = (i, j) if shells[i]["l"] >= shells[j]["l"] else (j, i)
            key = tuple((shells[x]["l"], shells[x]["spherical"]) for x in (a, b))
            by.setdefault(key, []).append((a, b))
    got = []
    for (ka, kb), pairs in by.items():
        ia = torch.tensor(np.array([off[a] + np.arange(_n_func(*ka)) for a, _ in pairs]), device=_dev())
        ib_ = torch.tensor(np.array([off[b] + np.arange(_n_func(*kb)) for _, b in pairs]), device=_dev())
        got.append((pairs, ia, ib_))
    return got


def _function_pairs(ia, ib_):
    """AO indices of the flattened functions of every pair: [n, na*nb]."""
    n = ia.shape[0]
    return (ia[:, :, None].expand(n, ia.shape[1], ib_.shape[1]).reshape(n, -1),
            ib_[:, None, :].expand(n, ia.shape[1], ib_.shape[1]).reshape(n, -1))


def _dense(shells, omega):
    """The whole tensor [nao, nao, nao, nao]."""
    n = _nao(shells)
    cls = _classes(shells)
    exp = [_pair_class(shells, pairs, False, False) for pairs, _, _ in cls]
    out = torch.zeros(n * n, n * n, dtype=torch.float64, device=_dev())
    fp = [_function_pairs(ia, ib_) for _, ia, ib_ in cls]
    for x in range(len(cls)):
        for y in range(x + 1):
            V = _blocks(exp[x], exp[y], omega)
            V = V.reshape(V.shape[0] * V.shape[1], -1)
            (a, b), (c, d) = [tuple(v.reshape(-1) for v in fp[k]) for k in (x, y)]
            for u, v in ((a, b), (b, a)):
                for w, z in ((c, d), (d, c)):
                    out[(u * n + v)[:, None], (w * n + z)[None, :]] = V
                    out[(w * n + z)[:, None], (u * n + v)[None, :]] = V.T
    return out.reshape(n, n, n, n)


def _exact_grad(shells, D, omega):
    """sum Gamma d(ij|kl)/dR with Gamma = D_ij D_kl / 2 - (D_ik D_jl + D_il D_jk) / 8:
    twice the derivative on the bra's centres, over every bra and ket."""
    atoms = list(dict.fromkeys(tuple(s["center"]) for s in shells))
    D = torch.from_numpy(np.ascontiguousarray(D)).to(_dev())
    g = torch.zeros(len(atoms), 3, dtype=torch.float64, device=_dev())
    cls = _classes(shells)
    ket = [_pair_class(shells, pairs, False, False) for pairs, _, _ in cls]
    fp = [_function_pairs(ia, ib_) for _, ia, ib_ in cls]
    for x, (pairs, _, _) in enumerate(cls):
        bra = _pair_class(shells, pairs, True, False)
        a, b = fp[x]
        wb = torch.tensor([1.0 if i == j else 2.0 for i, j in pairs], dtype=torch.float64, device=_dev())
        at = [torch.tensor([atoms.index(tuple(shells[p[w]]["center"])) for p in pairs], device=_dev()) for w in (0, 1)]
        for y, (kpairs, _, _) in enumerate(cls):
            c, d = fp[y]
            wk = torch.tensor([1.0 if i == j else 2.0 for i, j in kpairs], dtype=torch.float64, device=_dev())
            V = _blocks(bra, ket[y], omega)
            V = V.reshape(V.shape[0], 6, -1, V.shape[2], V.shape[3])
            a4, b4, c4, d4 = a[:, :, None, None], b[:, :, None, None], c[None, None], d[None, None]
            G = 0.5 * D[a4, b4] * D[c4, d4] - 0.125 * (D[a4, c4] * D[b4, d4] + D[a4, d4] * D[b4, c4])
            G = G * wb[:, None, None, None] * wk[None, None, :, None]
            s = 2.0 * torch.einsum("nsfmg,nfmg->ns", V, G)
            for w in (0, 1):
                g.index_add_(0, at[w], s[:, 3 * w:3 * w + 3])
    return g.cpu().numpy()


def _exact_df(shells, aux):
    n, na = _nao(shells), _nao(aux)
    off = np.cumsum([0] + [_n_func(s["l"], s["spherical"]) for s in aux])
    by = {}
    for i, s in enumerate(aux):
        by.setdefault((s["l"], s["spherical"], len(s["exps"])), []).append(i)
    ax = []
    for (l, sph, _), ids in by.items():
        e = _pair_class(aux, [(i, i) for i in ids], False, True)
        ax.append((e, torch.tensor(np.array([off[i] + np.arange(_n_func(l, sph)) for i in ids]), device=_dev()).reshape(-1)))
    t3 = torch.zeros(n, n, na, dtype=torch.float64, device=_dev())
    for pairs, ia, ib_ in _classes(shells):
        e = _pair_class(shells, pairs, False, False)
        a, b = (v.reshape(-1) for v in _function_pairs(ia, ib_))
        for ek, at in ax:
            V = _blocks(e, ek, 0.0).reshape(len(a), -1)
            t3[a[:, None], b[:, None], at[None]] = V
            t3[b[:, None], a[:, None], at[None]] = V
    t2 = torch.zeros(na, na, dtype=torch.float64, device=_dev())
    for e, at in ax:
        for ek, kt in ax:
            t2[at[:, None], kt[None]] = _blocks(e, ek, 0.0).reshape(len(at), -1)
    return t3.reshape(-1).cpu().numpy(), t2.reshape(-1).cpu().numpy()


def _exact_cost(shells, deriv):
    cost = 0.0
    cls = {}
    for s in shells:
        cls.setdefault((s["l"], len(s["exps"])), []).append(s)
    per = []
    for (la, ka), u in cls.items():
        for (lb, kb), v in cls.items():
            if la >= lb:
                per.append((len(u) * len(v) * (0.5 if la == lb else 1.0) * ka * kb, math.comb(la + lb + 3 + deriv, 3)))
    for n, h in per:
        for m, k in per:
            cost += 0.5 * n * m * h * k * (8.0 if deriv else 2.0)
    return cost


def exact(case, seed):
    inp = _inputs(case, seed)
    op = case["op"]
    mols = inp["molecules"] if op == "batch" else [inp["shells"]]
    cost = sum(_exact_cost(m, op in ("grad", "batch")) for m in mols)
    if case["share"] != 1 or (op != "df" and (cost > 4e11 or max(_nao(m) for m in mols) > 128)):
        return None
    if op == "df":
        t3, t2 = _exact_df(inp["shells"], inp["aux"])
        return {"eri_3c": t3, "eri_2c": t2}
    if op == "grad":
        return {"grad": _exact_grad(inp["shells"], inp["dens"], case["omega"])}
    if op in ("jk", "jk_host"):
        V = _dense(inp["shells"], 0.0)
        D = torch.from_numpy(inp["dens"]).to(_dev())
        J = torch.einsum("ijkl,xkl->xij", V, D)
        K = torch.einsum("ikjl,xkl->xij", V, D) if case["exchange"] else None
        return {"J": J.cpu().numpy(), "K": None if K is None else K.cpu().numpy()}
    if op in ("eri", "rows"):
        return {"eri": _dense(inp["shells"], case["omega"]).reshape(-1).cpu().numpy()}
    if op == "packed":
        shells = inp["shells"]
        V = _dense(shells, 0.0)
        off = np.cumsum([0] + [_n_func(s["l"], s["spherical"]) for s in shells])
        ao = [(off[i] + a, off[j] + b) for i in range(len(shells)) for j in range(i + 1)
              for a in range(off[i + 1] - off[i]) for b in range(a + 1 if i == j else off[j + 1] - off[j])]
        ao = torch.tensor(np.array(ao), device=_dev())
        t, u = torch.tril_indices(len(ao), len(ao), device=_dev())
        return {"eri": V[ao[t, 0], ao[t, 1], ao[u, 0], ao[u, 1]].cpu().numpy()}
    got = {"J": [], "K": [], "grad": []}
    for shells, D in zip(inp["molecules"], inp["dens"]):
        V = _dense(shells, 0.0)
        d = torch.from_numpy(D).to(_dev())
        got["J"].append(torch.einsum("ijkl,kl->ij", V, d).reshape(-1).cpu().numpy())
        got["K"].append(torch.einsum("ikjl,kl->ij", V, d).reshape(-1).cpu().numpy())
        got["grad"].append(_exact_grad(shells, D, 0.0))
    return {k: np.concatenate(v) for k, v in got.items()}
