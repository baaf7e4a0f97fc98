"""The work a user of this framework has it do, as measurable cases.

Five kinds of call, all through the package's public entry points:

  product  y = T x on device vectors (TMatOp.perform_op_dev), the call every
           Krylov solver makes, in FP32, FP64 or double-float (TM_F64_DF)
  eigs     a solve on an operator the program already holds (TMatOp.eigs)
  solve    one parameter point from nothing: operator, eigenvalues, close
  grad     the adjoint: d ln(lambda) / d(betaJ, kappa, kappa2, h)
  sweep    a batch of parameter points solved together (Sweep.eigs)

Sizes and parameters are those of the repository's configurations and parity
fixtures.  A product state holds its operator and vectors; a solve or sweep
starts from the parameter points alone, as the tmat driver does.
"""
import math

import numpy as np
import torch

import latttmat_gb300 as lt

DTYPES = {"f64": lt.TM_F64, "f32": lt.TM_F32, "df": lt.TM_F64_DF}

# (model, dim, axialdir) -> default parameters (betaJ, kappa, kappa2, h)
POINTS = {
    ("A", 2, 1): (0.5, 0.5, 0.0, 0.0), ("A", 2, 5): (0.3, 0.6, 0.0, 0.0), ("A", 3, 1): (0.2, 0.4, 0.0, 0.0),
    ("A", 2, 2): (0.3, 0.6, 0.0, 0.0), ("A", 2, 0): (0.3, 0.6, 0.0, 0.0), ("A", 2, 6): (0.3, 0.6, 0.0, 0.0),
    ("D", 2, 2): (0.4, 0.3, 0.0, 0.1), ("D", 2, 5): (0.4, 0.3, 0.0, 0.0),
    ("B", 2, 3): (0.5, 0.6, 0.2, 0.0), ("B", 2, 7): (0.6, 0.8, 0.0, 0.0), ("B", 2, 6): (0.5, 0.3, 0.2, 0.0),
}
REDUCED = {("A", 2, 5), ("A", 3, 1), ("D", 2, 5), ("B", 2, 7), ("A", 2, 6), ("B", 2, 6)}
TWO_LAYER = {("A", 2, 2), ("A", 2, 0), ("A", 2, 6), ("B", 2, 6)}


def _case(kind, model, dim, axialdir, size1, size2=0, **more):
    bj, k, k2, h = POINTS[(model, dim, axialdir)]
    c = {"kind": kind, "model": model, "dim": dim, "axialdir": axialdir, "size1": size1, "size2": size2,
         "betaJ": bj, "kappa": k, "kappa2": k2, "h": h, "extend_cond": 2, "transpose": False, "dtype": "f64"}
    c.update(more)
    return c


def listed():
    named = [
        # a product on the smallest operator in the configurations: latency
        ("product_xat_L12_f64", _case("product", "A", 2, 1, 12)),
        # a whole solve with eigenvectors at that end, as one tmat run does
        ("eigs_xat_L14_f64", _case("eigs", "A", 2, 1, 14, betaJ=0.9, kappa=0.2, h=0.05, nev=2, tol=1e-12)),
        # the headline operator, FP32 products of its Lanczos phase
        ("product_xam_L32_f32", _case("product", "A", 2, 5, 32, dtype="f32")),
        # FP64-accurate products of its refinement
        ("product_xam_L30_df", _case("product", "A", 2, 5, 30, dtype="df")),
        # the same reduced operator at an odd width, in FP64
        ("product_xam_L25_f64", _case("product", "A", 2, 5, 25)),
        # the full DNNI operator with 6.7e7 states, FP32
        ("product_xdt_L26_f32", _case("product", "D", 2, 2, 26, dtype="f32")),
        # the widest operator of the BNNNI sweep, FP64-accurate products
        ("product_zbm_L24_df", _case("product", "B", 2, 7, 24, dtype="df")),
        # the 3D operator on a 5x5 layer, FP64
        ("product_x3d_5x5_f64", _case("product", "A", 3, 1, 5, 5, extend_cond=0)),
        # a two-layer parallel operator with 2^24 states, FP64
        ("product_yat_L12_f64", _case("product", "A", 2, 2, 12)),
        # the adjoint of the reduced operator at the gradient workload's width
        ("grad_xam_L24", _case("grad", "A", 2, 5, 24, betaJ=0.35, kappa=0.55, h=0.05, extend_cond=0)),
        # a parameter sweep of mixed widths, all points as one device batch
        ("sweep_zbm_16pt", _case("sweep", "B", 2, 7, 22, points=16, nev=2, tol=1e-10)),
        # one point of the headline workload, construction to eigenvalues
        ("solve_xam_L32_mixed", _case("solve", "A", 2, 5, 32, dtype="mixed", nev=4, tol=1e-10)),
    ]
    return [dict(c, name=n) for n, c in named]


def draw(rng):
    kind = rng.choice(["product"] * 8 + ["eigs", "solve", "grad", "grad", "sweep"])
    bj, k = round(rng.uniform(0.2, 0.9), 3), round(rng.uniform(0.0, 1.0), 3)
    h = rng.choice([0.0, 0.0, 0.05, 0.1])
    if kind == "sweep":
        return _case("sweep", "B", 2, 7, rng.choice([16, 18, 20, 22]), points=rng.randint(3, 16), nev=2, tol=1e-10)
    if kind in ("eigs", "solve"):
        model, dim, ax, lo, hi = rng.choice([("A", 2, 1, 10, 18), ("A", 2, 5, 12, 30), ("D", 2, 5, 10, 18)])
        return _case(kind, model, dim, ax, rng.randint(lo, hi), betaJ=round(rng.uniform(0.2, 0.5), 3),
                     kappa=round(rng.uniform(0.0, 0.4), 3), h=0.05, dtype=rng.choice(["f64", "mixed"]), nev=2,
                     tol=1e-12)
    if kind == "grad":
        model, dim, ax, lo, hi = rng.choice([("A", 2, 1, 10, 20), ("A", 2, 5, 12, 24), ("D", 2, 5, 10, 20),
                                             ("B", 2, 7, 10, 20), ("A", 3, 1, 3, 5)])
        s1 = rng.randint(lo, hi)
        if model == "B":
            s1 -= s1 % 2
        return _case("grad", model, dim, ax, s1, rng.randint(3, 5) if dim == 3 else 0, betaJ=bj, kappa=k, h=h,
                     kappa2=0.1 if model == "B" else 0.0, extend_cond=rng.choice([0, 2]) if dim == 2 else 0)
    model, dim, ax, lo, hi = rng.choice([
        ("A", 2, 1, 8, 26), ("A", 2, 5, 10, 31), ("A", 2, 5, 12, 31), ("A", 3, 1, 3, 5), ("D", 2, 2, 8, 25),
        ("D", 2, 5, 10, 25), ("B", 2, 3, 8, 22), ("B", 2, 7, 12, 24), ("A", 2, 2, 4, 13), ("A", 2, 0, 4, 12),
        ("A", 2, 6, 5, 13), ("B", 2, 6, 5, 12)])
    s1 = rng.randint(lo, hi)
    if model == "B" and ax != 6:
        s1 -= s1 % 2
    dtype = "f64" if (model, dim, ax) in TWO_LAYER else rng.choice(["f64", "f32", "df"])
    turned = (model == "B" or (model, dim, ax) in TWO_LAYER) and rng.random() < 0.4
    return _case("product", model, dim, ax, s1, rng.randint(3, 5) if dim == 3 else 0, betaJ=bj, kappa=k, h=h,
                 kappa2=0.1 if model == "B" else 0.0, dtype=dtype, transpose=turned,
                 extend_cond=rng.choice([0, 2]) if dim == 2 else 0)


# ------------------------------------------------------------------ a user's program
def _key(c):
    return (c["model"], c["dim"], c["axialdir"])


def _operator(c):
    size = (c["size1"], c["size2"]) if c["dim"] == 3 else c["size1"]
    return lt.TMatOp(c["model"], c["dim"], c["axialdir"], c["betaJ"], c["kappa"], c["h"], size, c["kappa2"],
                     c["extend_cond"])


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _vector(n, seed):
    """A Krylov vector: unit norm, components of both signs."""
    x = torch.randn(n, generator=_generator(seed), device="cuda", dtype=torch.float64)
    return x / x.norm()


def _positive(n, seed):
    """A Perron-like vector: positive, unit norm."""
    x = torch.rand(n, generator=_generator(seed), device="cuda", dtype=torch.float64) + 0.5
    return x / x.norm()


def _point(c, seed):
    """The case's parameters at a point near its own, one per seed."""
    u = np.random.default_rng(seed).uniform(-1.0, 1.0, 2)
    return dict(c, betaJ=c["betaJ"] * (1.0 + 0.01 * u[0]), kappa=c["kappa"] * (1.0 + 0.01 * u[1]))


def _sweep_points(c, seed):
    """Widths in equal shares up to the case's, betaJ on a grid over [0.2, 1.0], kappa uniform."""
    r = np.random.default_rng(seed)
    widths = [w for w in (16, 18, 20, 22, 24) if w <= c["size1"]]
    bj = np.linspace(0.2, 1.0, c["points"])
    return [(float(bj[i]), float(r.uniform(0.0, 1.0)), 0.0, 0.0, widths[i % len(widths)]) for i in range(c["points"])]


GRAD_LAMBDA = 0.7  # reported eigenvalue the gradient is formed with (it only scales one term)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    if kind == "product":
        op = _operator(case)
        use = op.get_t_instance() if case["transpose"] else op
        x = _vector(op.rows(), seed)
        s.update(base=op, op=use, dtype=DTYPES[case["dtype"]], stream=torch.cuda.Stream(),
                 x=x.float() if case["dtype"] == "f32" else x)
        s["y"] = torch.empty_like(s["x"])
        torch.cuda.synchronize()
    elif kind == "eigs":
        s["op"] = _operator(_point(case, seed))
    elif kind == "solve":
        s["point"] = _point(case, seed)
    elif kind == "grad":
        s["op"] = _operator(case)
        n = s["op"].rows()
        s["qr"] = _positive(n, seed).cpu().numpy()
        s["ql"] = None if s["op"].is_symmetric() else _positive(n, seed + 1).cpu().numpy()
        s["lam"] = GRAD_LAMBDA * s["op"].getnormfactor()
    else:
        s["points"] = _sweep_points(case, seed)
    return s


def _mode(c):
    return lt.TM_EIGS_MIXED if c["dtype"] == "mixed" else lt.TM_EIGS_F64


def run(state):
    c, kind = state["case"], state["kind"]
    if kind == "product":
        state["op"].perform_op_dev(state["x"].data_ptr(), state["y"].data_ptr(), state["dtype"],
                                   state["stream"].cuda_stream)
        return state["y"]
    if kind == "eigs":
        vals, vecs, _, _ = state["op"].eigs(c["nev"], tol=c["tol"], mode=_mode(c), vectors=True)
        return [vals, vecs]
    if kind == "solve":
        op = _operator(state["point"])
        vals, _, _, _ = op.eigs(c["nev"], tol=c["tol"], mode=_mode(c))
        op.close()
        return vals
    if kind == "grad":
        return state["op"].grad(state["qr"], state["lam"], state["ql"])
    sweep = lt.Sweep(c["model"], c["dim"], c["axialdir"], state["points"], c["extend_cond"])
    vals, _, _ = sweep.eigs(nev=c["nev"], tol=c["tol"], mode=lt.TM_EIGS_MIXED)
    sweep.close()
    return vals


# ------------------------------------------------------------------ what a pass cannot do without
def _bits(c):
    if c["dim"] == 3:
        return c["size1"] * c["size2"]
    return 2 * c["size1"] if _key(c) in TWO_LAYER else c["size1"]


def _flip(c):
    if _key(c) not in REDUCED:
        return False
    return c["h"] == 0.0 and (c["dim"] == 3 or not c["extend_cond"] & 2)


def _rows(c):
    """Length of the operator's vectors (reduced: states over the group's order)."""
    n = 1 << _bits(c)
    if _key(c) not in REDUCED:
        return n
    order = 4 * c["size1"] * c["size2"] if c["dim"] == 3 else (c["size1"] if _key(c) == ("B", 2, 7) else 2 * c["size1"])
    return max(1, n // (order * (2 if _flip(c) else 1)))


def work(case):
    """Each vector read or written once; one multiply-add per site and row of
    a product.  A solve: the products and basis vectors of a Krylov space of
    30 columns; a gradient: one product per parameter its gates depend on."""
    n, L = _rows(case), _bits(case)
    kind = case["kind"]
    item = 4 if case["dtype"] == "f32" else 8
    if kind == "product":
        return {"bytes": 2 * n * item, "flops": 2 * L * n}
    if kind == "grad":
        return {"bytes": 2 * n * 8, "flops": 3 * 2 * L * n}
    item = 4 if case["dtype"] == "mixed" else 8
    if kind == "sweep":
        rows = sum(_rows(dict(case, size1=w)) for _, _, _, _, w in _sweep_points(case, 0))
        return {"bytes": 25 * 3 * rows * 4, "flops": 25 * 2 * L * rows}
    return {"bytes": 30 * 3 * n * item, "flops": 30 * 2 * L * n}


# ------------------------------------------------------------------ the same in 64 bits, plain torch
def _popc(v):
    v = v - ((v >> 1) & 0x5555555555555555)
    v = (v & 0x3333333333333333) + ((v >> 2) & 0x3333333333333333)
    v = (v + (v >> 4)) & 0x0F0F0F0F0F0F0F0F
    v = v + (v >> 8)
    v = v + (v >> 16)
    return (v + (v >> 32)) & 127


def _rotr(s, L, d):
    d %= L
    return (s >> d) | ((s & ((1 << d) - 1)) << (L - d)) if d else s


def _brev(s, L):
    r = torch.zeros_like(s)
    for i in range(L):
        r |= ((s >> i) & 1) << (L - 1 - i)
    return r


def _images(c, s):
    """All images of the states s under the operator's layer group (flip left out)."""
    L = c["size1"]
    if c["dim"] == 3:
        rows, cols = c["size1"], c["size2"]
        n = rows * cols
        low = sum(1 << (r * cols) for r in range(rows))  # column 0 of every row
        permuted = []
        for mr in (0, 1):
            for mc in (0, 1):
                t = torch.zeros_like(s)
                for r in range(rows):
                    for q in range(cols):
                        to = (rows - 1 - r if mr else r) * cols + (cols - 1 - q if mc else q)
                        t |= ((s >> (r * cols + q)) & 1) << to
                permuted.append(t)
        if c["kappa"] == 0.0 and rows == cols:  # quarter turns, in the isotropic case
            for base in list(permuted):
                t = torch.zeros_like(s)
                for r in range(rows):
                    for q in range(cols):
                        t |= ((base >> (r * cols + q)) & 1) << ((q + 1) * cols - (r + 1))
                permuted.append(t)
        for t in permuted:
            for _ in range(cols):
                u = t
                for _ in range(rows):
                    yield u
                    u = _rotr(u, n, cols)
                t = ((t >> 1) & ~(low << (cols - 1))) | ((t & low) << (cols - 1))
    elif _key(c) == ("B", 2, 7):
        r = _brev(_rotr(s, L, 1), L)
        for d in range(0, L, 2):
            yield _rotr(s, L, d)
            yield _rotr(r, L, d)
    elif _key(c) in TWO_LAYER:
        m = (1 << L) - 1
        hi, lo = s >> L, s & m
        bh, bl = _brev(hi, L), _brev(lo, L)
        for d in range(L):
            yield (_rotr(hi, L, d) << L) | _rotr(lo, L, d)
            yield (_rotr(bh, L, d) << L) | _rotr(bl, L, d)
    else:
        b = _brev(s, L)
        for d in range(L):
            yield _rotr(s, L, d)
            yield _rotr(b, L, d)


def _orbits(c):
    """(rank of every state's orbit, representatives ascending, orbit sizes)."""
    nb = _bits(c)
    s = torch.arange(1 << nb, device="cuda", dtype=torch.int64)
    best = s.clone()
    for im in _images(c, s):
        torch.minimum(best, im, out=best)
        if _flip(c):
            torch.minimum(best, im ^ ((1 << nb) - 1), out=best)
    reps = s[best == s]
    rank = torch.searchsorted(reps, best)
    return rank, reps, torch.bincount(rank, minlength=len(reps))


def _nfexp(c):
    k, k2, L = c["kappa"], c["kappa2"], c["size1"]
    if c["model"] == "B":
        if k + k2 < 0.5:
            return L * 2.0 * (k + k2 - 1.0)
        if k < 0.5 and k2 - k < 0.5:
            return -L
        return -L * 2.0 * k if k2 < 2 * k else L * 2.0 * (k - k2)
    if c["model"] == "D":
        return L * 2.0 * (k - 1.0) if k < 0.5 else -L * 2.0 * k
    if c["dim"] == 3:
        L = _bits(c)
        return L * (k - 3.0) if k < 0.5 else -L * (k + 2.0)
    if c["axialdir"] == 0:
        return 2 * L * (k - 2.0) if k < 0.5 else -2 * L * (k + 1.0)
    return L * (k - 2.0) if k < 0.5 else -L * (k + 1.0)


def _weights(c, s):
    """(ln Tvec without the normfactor, its derivatives by betaJ, kappa, kappa2, h) of the states s."""
    K, k, k2, h, L = c["betaJ"], c["kappa"], c["kappa2"], c["h"], c["size1"]
    f = torch.float64
    if _key(c) in TWO_LAYER:
        m = (1 << L) - 1
        lo, hi = s & m, s >> L
        if c["axialdir"] == 2:
            n1, n0, nx = _popc(lo ^ _rotr(lo, L, 1)), _popc(lo), _popc(lo ^ hi)
            return (-K * ((2 * (n1 + nx) - 2 * L).to(f) + h * (2 * n0 - L).to(f)), None)
        if c["axialdir"] == 0:
            bonds = _popc(lo ^ _rotr(lo, L, 1)) + _popc(hi ^ _rotr(hi, L, 1)) + _popc(lo ^ hi)
            return (-0.5 * K * ((2 * bonds - 3 * L).to(f) + 2 * h * (_popc(s) - L).to(f)), None)
        n1 = _popc(hi ^ _rotr(hi, L, 1)) + _popc(hi ^ lo)
        w = -0.5 * K * ((2 * (n1 - L)).to(f) + h * (2 * _popc(hi) - L).to(f))
        if c["model"] == "B":
            d = _popc(hi ^ _rotr(lo, L, 1)) + _popc(hi ^ _rotr(lo, L, L - 1))
            w = w + 0.5 * K * (k * (2 * _popc(hi ^ _rotr(hi, L, 2)) - L).to(f) + k2 * (2 * (d - L)).to(f))
        return (w, None)
    n = _bits(c)
    zero = torch.zeros((), dtype=f, device=s.device)
    field = (2 * _popc(s) - n).to(f)
    if c["dim"] == 3:
        rows, cols = c["size1"], c["size2"]
        low = sum(1 << (r * cols) for r in range(rows))

        def right(v, d):
            for _ in range(d):
                v = ((v >> 1) & ~(low << (cols - 1))) | ((v & low) << (cols - 1))
            return v

        near = 2.0 * (_popc(s ^ right(s, 1)) + _popc(s ^ _rotr(s, n, cols)) - n).to(f)
        nextn = (2 * _popc(s ^ right(s, 2)) - n).to(f)
    else:
        near = (2 * _popc(s ^ _rotr(s, L, 1)) - L).to(f)
        nextn = (2 * _popc(s ^ _rotr(s, L, 2)) - L).to(f)
    frus = {"A": k, "B": k2, "D": 0.0}[c["model"]]
    per_k = -0.5 * near + 0.5 * frus * nextn - 0.5 * h * field
    by_frus = 0.5 * K * nextn
    grads = [per_k, by_frus if c["model"] == "A" else zero, by_frus if c["model"] == "B" else zero, -0.5 * K * field]
    return (K * per_k, grads)


def _kron(v, lo, hi, a, b):
    """[[a, b], [b, a]] on bits [lo, hi)."""
    for i in range(lo, hi):
        x = v.view(-1, 2, 1 << i)
        x0, x1 = x[:, 0], x[:, 1]
        v = torch.stack((a * x0 + b * x1, b * x0 + a * x1), 1).view(-1)
    return v


def _gates(c, K, k, k2, transpose):
    """w[s', q], u[s', a'], z[f, s'] of one step of the site-by-site product."""
    e = [torch.exp(t) for t in (K, -K * k, -K * k2)]
    b1, b2, b3 = [[x, 1.0 / x] for x in e]
    if c["model"] == "D":
        return ([[b2[s ^ q] for q in (0, 1)] for s in (0, 1)], [[b1[s ^ a] for a in (0, 1)] for s in (0, 1)],
                [[b2[f ^ s] for s in (0, 1)] for f in (0, 1)])
    w, u, z = ([[None] * 4 for _ in range(4)] for _ in range(3))
    for x in range(4):
        xl, xr = x >> 1, x & 1
        for y in range(4):
            yl, yr = y >> 1, y & 1
            w[x][y] = b2[xr ^ yr] * b2[xl ^ yl] * (1.0 if transpose else b1[xr ^ yl])
            u[x][y] = b3[xr ^ yr] * b3[xl ^ yl] * (b1[xl ^ yr] if transpose else b1[xr ^ yl])
            z[x][y] = b2[yr ^ xr] * b2[yl ^ xl] * (b1[yl ^ xr] if transpose else 1.0)
    return w, u, z


def _chain(c, v, K, k, k2, transpose):
    """The inter-layer factor of the DNNI and diagonal BNNNI operators on a full vector."""
    L, S, bits = c["size1"], 2 if c["model"] == "D" else 4, 1 if c["model"] == "D" else 2
    w, u, z = (torch.stack([torch.stack(list(r)) for r in t]) for t in _gates(c, K, k, k2, transpose))
    total = 0.0
    for first in range(S):
        # every new site needs the old sites on both sides: the ring is cut at its first old site
        cut = v.view(-1, S).clone()
        cut[:, [q for q in range(S) if q != first]] = 0
        cut = cut.view(S, -1)  # by the last old site, which the first step sees as its left neighbour
        t = torch.zeros((S,) + (v.numel(),), dtype=v.dtype, device=v.device).view(S, S, -1)
        for q in range(S):
            t[q, q] = cut[q]
        for step in range(L // bits):
            low = S ** step
            if step < L // bits - 1:
                x = t.reshape(S, -1, S, S, low)  # carried, rest, next old site, old site, new sites below
                out = torch.empty_like(x)
                for a in range(S):
                    for s in range(S):
                        d = sum(w[s, q] * x[q, :, :, a] for q in range(S))
                        out[a, :, :, s] = u[s, a] * z[:, s].view(1, S, 1) * d
            else:
                x = t.reshape(S, S, low)
                out = torch.empty_like(x)
                for a in range(S):
                    for s in range(S):
                        out[a, s] = u[s, a] * z[first, s] * sum(w[s, q] * x[q, a] for q in range(S))
            t = out
        total = total + t.reshape(S, -1).sum(0)
    return total


def _core(c, v, transpose, shift=None):
    """The inter-layer factor on a full vector; `shift`: complex steps of (betaJ, kappa, kappa2)."""
    step = shift or (0.0, 0.0, 0.0)
    kind = torch.complex128 if shift else torch.float64
    K, k, k2 = (torch.tensor(c[p] + d, dtype=kind, device=v.device) for p, d in zip(("betaJ", "kappa", "kappa2"), step))
    if shift:
        v = v.to(kind)
    if c["model"] == "A":
        return _kron(v, 0, _bits(c), torch.exp(K), torch.exp(-K))
    return _chain(c, v, K, k, k2, transpose)


class _Exact:
    """The operator's product in 64 bits, from its definition."""

    def __init__(self, c):
        self.c, self.reduced = c, _key(c) in REDUCED
        nb = _bits(c)
        self.nf = math.exp(c["betaJ"] * _nfexp(c))
        if self.reduced:
            self.rank, self.states, self.dup = _orbits(c)
        else:
            self.states = torch.arange(1 << nb, device="cuda", dtype=torch.int64)
        lnw, self.grads = _weights(c, self.states)
        self.tv = torch.exp(lnw)
        if self.reduced:
            # (the y-direction operators without the half normfactor of the others are the full ones)
            self.tv = self.tv * math.sqrt(self.nf) / torch.sqrt(self.dup.double())

    def spread(self, x):
        x = self.tv * x
        return x[self.rank] if self.reduced else x

    def collect(self, z):
        return self.tv * self.dup * z[self.states] if self.reduced else self.tv * z * self.nf

    def product(self, x):
        c, turned, L = self.c, self.c["transpose"], self.c["size1"]
        if _key(c) not in TWO_LAYER:
            return self.collect(_core(c, self.spread(x), turned))
        K, k = c["betaJ"], c["kappa"]
        w0, w1 = math.exp(-K * k), math.exp(K * k)
        N = 1 << L

        def swap(v):
            return v.view(N, N).t().reshape(-1)

        if c["axialdir"] == 2:
            if turned:
                return self.nf * swap(_kron(self.tv * x, 0, L, w0, w1))
            return self.nf * self.tv * swap(_kron(x, L, 2 * L, w0, w1))
        if c["axialdir"] == 0:
            v = self.tv * x
            e1, e2 = (math.exp(K), math.exp(-K)), (math.exp(-2 * K * k), math.exp(2 * K * k))
            for i in range(L):
                t = v.view(1 << (L - 1 - i), 2, 1 << (L - 1), 2, 1 << i)  # the bit pair (i, L + i)
                out = torch.empty_like(t)
                for hi in (0, 1):
                    for lo in (0, 1):
                        j = lo ^ hi
                        out[:, hi, :, lo] = (e1[j] * (e2[0] * t[:, hi, :, lo] + t[:, 1 - hi, :, lo])
                                             + e1[1 - j] * (e2[1] * t[:, 1 - hi, :, 1 - lo] + t[:, hi, :, 1 - lo]))
                v = out.view(-1)
            return self.nf * self.tv * v
        u = (self.tv * x)[self.rank]
        if turned:
            return self.tv * self.dup * _kron(swap(u), 0, L, w0, w1)[self.states]
        return self.tv * self.dup * swap(_kron(u, 0, L, w0, w1))[self.states]


def _exact_values(c, nev):
    """The leading eigenvalues of a symmetric operator, by Lanczos with full reorthogonalisation."""
    T = _Exact(c)
    n = len(T.states)
    m = min(n, 90)
    V = torch.zeros(m + 1, n, dtype=torch.float64, device="cuda")
    V[0] = _positive(n, 1)
    H = np.zeros((m, m))
    for j in range(m):
        w = T.product(V[j])
        for again in (0, 1):
            d = V[: j + 1] @ w
            w = w - d @ V[: j + 1]
            if not again:
                H[: j + 1, j] = d.cpu().numpy()
                H[j, : j + 1] = H[: j + 1, j]
        b = float(w.norm())
        if b < 1e-14 * abs(H[0, 0]):
            H = H[: j + 1, : j + 1]
            break
        V[j + 1] = w / b
    vals = np.linalg.eigvalsh(H)
    return vals[np.argsort(-np.abs(vals))][:nev] / T.nf


def exact(case, seed):
    kind = case["kind"]
    if kind == "sweep" or _bits(case) > 28:
        return None
    if kind in ("eigs", "solve"):
        if _bits(case) > 20:
            return None
        vals = _exact_values(_point(case, seed), case["nev"])
        return [vals, None] if kind == "eigs" else vals
    T = _Exact(case)
    n = len(T.states)
    if kind == "product":
        x = _vector(n, seed)
        return T.product((x.float() if case["dtype"] == "f32" else x).double())
    r = _positive(n, seed)
    left = r if case["model"] != "B" else _positive(n, seed + 1)
    lr = left * r
    total = lr.sum()
    lam = GRAD_LAMBDA * T.nf
    out = [float(2.0 * (lr * g).sum() / total) for g in T.grads]
    size = 1e-20
    for i in range(1 if case["model"] == "A" else (3 if case["model"] == "B" else 2)):
        step = [0.0, 0.0, 0.0]
        step[i] = 1j * size
        d = _core(case, T.spread(r), False, tuple(step)).imag / size
        out[i] += float((left * T.collect(d)).sum() / (lam * total))
    return np.array(out)
