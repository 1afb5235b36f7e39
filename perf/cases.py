"""The solves that a user of this package runs, as cases to be timed.

Every case is one call of a public entry point with what a program has in hand before it: sparse
operators created once from CSR arrays, random-phase states and result buffers on the device (or,
for the post-processor of a moment file, the table on the host).  The operators are seeded
tight-binding lattices with Anderson disorder, already rescaled to the Chebyshev domain.

    dos             linqt_moments1d_dev: density of states, or a spectral operator <r|T_m(H) V|r>
    realisations    linqt_moments1d_realisations_dev: a DOS averaged over disorder seeds
    moments2d       linqt_moments2d_dev: the correlation table <r|V T_m(H) V T_n(H)|r>
    kubo_bastin     linqt_kubo_bastin_dev: that table and sigma(E) from one recursion
    kubo_greenwood  linqt_kubo_fft_dev with the Greenwood formula: sigma(E) alone
    time            linqt_moments_td_dev: time-domain correlations
    post_bastin     linqt_bastin_from_moments: sigma(E) from a moment table on the host
"""
import math

import numpy as np
import torch

import linqt_b200 as lq

HBAR = 0.6582119624  # eV fs, the constant of the time-correlation interface


# ---------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------
def _case(name, kind, lattice, dims, R, M, **more):
    lx, ly, lz = tuple(dims) + (1,) * (3 - len(dims))
    c = {"kind": kind, "lattice": lattice, "lx": lx, "ly": ly, "lz": lz, "R": R, "M": M, "mixed": False}
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: a quick look at a few hundred sites with one vector, bound by latency
        _case("dos_square_31", "dos", "square", (31, 31), 1, 100, velocity=False),
        # a plain DOS of a 2D lattice, one vector, many moments: hundreds of short dependent steps
        _case("dos_square_256", "dos", "square", (256, 256), 1, 1024, velocity=False),
        # a spectral operator (no doubling of the moments) with an odd number of vectors and moments
        _case("spectral_op_graphene_97x64", "dos", "honeycomb", (97, 64), 5, 301, velocity=True),
        # a wide block of vectors on a 3D lattice far larger than the caches
        _case("dos_cubic_100_r64", "dos", "cubic", (100, 100, 100), 64, 128, velocity=False),
        # disorder average: 4 seeds of a 3D lattice, 8 vectors each, FP32 vectors, one launch
        _case("realisations_cubic_40", "realisations", "cubic", (40, 40, 40), 32, 512, seeds=4, mixed=True),
        # the smallest correlation table: one vector and the 100 moments of a first run
        _case("moments2d_graphene_20", "moments2d", "honeycomb", (20, 20), 1, 100),
        # spin-transport table, Kane-Mele, FP64: the contraction of 1024 moments of 32 vectors
        _case("moments2d_kane_mele_64", "moments2d", "kane_mele", (64, 64), 32, 1024),
        # the whole Kubo-Bastin solve at the benchmark's size, FP64
        _case("kubo_bastin_graphene_128", "kubo_bastin", "honeycomb", (128, 128), 8, 512, nump=1024),
        # the whole solve in mixed precision on the spin model
        _case("kubo_bastin_mixed_km_64", "kubo_bastin", "kane_mele", (64, 64), 16, 512, nump=1024, mixed=True),
        # Greenwood conductivity with a ragged number of vectors, moments and energies
        _case("greenwood_graphene_48x40", "kubo_greenwood", "honeycomb", (48, 40), 3, 300, nump=1000),
        # time-dependent velocity correlations: a 1D recursion and two evolutions per time step
        _case("time_corr_graphene_64", "time", "honeycomb", (64, 64), 4, 256, steps=8),
        # the post-processor of a moment file: 30 energies per moment
        _case("post_bastin_512", "post_bastin", "none", (1, 1), 1, 512, sites=32768),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, lattice, sites):
    """Extents (at least 3 cells) of a lattice of about `sites` sites, unequal and often odd."""
    if lattice == "cubic":
        e = sites ** (1 / 3)
        return tuple(max(3, int(round(e * rng.uniform(0.8, 1.25)))) for _ in range(3))
    cells = sites / {"square": 1, "honeycomb": 2, "kane_mele": 4}[lattice]
    lx = max(3, int(round(math.sqrt(cells) * rng.uniform(0.7, 1.4))))
    return lx, max(3, int(round(cells / lx)))


def draw(rng):
    kind = rng.choice(["dos", "dos", "realisations", "moments2d", "moments2d", "kubo_bastin", "kubo_bastin",
                       "kubo_greenwood", "time", "post_bastin"])
    if kind == "dos":
        lattice = rng.choice(["square", "cubic", "honeycomb", "kane_mele"])
        sites, R, M = _log(rng, 500, 600000), _log(rng, 1, 64), _log(rng, 64, 1024)
        while sites * R * M > 4e9:  # no dearer than the listed 3D lattice
            R, M = max(1, R // 2), max(64, M // 2)
            if R == 1 and M == 64:
                break
        velocity = lattice in ("honeycomb", "kane_mele") and rng.random() < 0.5
        return _case(None, kind, lattice, _dims(rng, lattice, sites), R, M, velocity=velocity, mixed=rng.random() < 0.3)
    if kind == "realisations":
        seeds, each = rng.randint(2, 4), 2 ** rng.randint(0, 3)
        return _case(None, kind, "cubic", _dims(rng, "cubic", _log(rng, 1000, 64000)), seeds * each,
                     _log(rng, 64, 512), seeds=seeds, mixed=rng.random() < 0.5)
    if kind == "post_bastin":
        return _case(None, kind, "none", (1, 1), 1, _log(rng, 50, 600), sites=_log(rng, 500, 1000000))
    lattice = rng.choice(["honeycomb", "kane_mele"])
    if kind == "time":
        return _case(None, kind, lattice, _dims(rng, lattice, _log(rng, 500, 20000)), _log(rng, 1, 8),
                     _log(rng, 64, 300), steps=rng.randint(2, 10))
    sites, R, M = _log(rng, 500, 40000), _log(rng, 1, 32), _log(rng, 64, 1024)
    while float(M) * M * sites * R > 2e11:  # no dearer than the listed spin-transport table
        R, M = max(1, R // 2), max(64, (2 * M) // 3)
        if R == 1 and M == 64:
            break
    if kind == "moments2d":
        return _case(None, kind, lattice, _dims(rng, lattice, sites), R, M, mixed=rng.random() < 0.3)
    fast = [n for n in (256, 512, 1024) if n >= M]
    nump = rng.choice(fast)
    if rng.random() < 0.3 and sites * R <= 20000 and M <= 400:  # any number of energies is taken
        nump = rng.randint(M, 2 * M + 200)
    return _case(None, kind, lattice, _dims(rng, lattice, sites), R, M, nump=nump,
                 mixed=kind == "kubo_bastin" and rng.random() < 0.4)


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
def _lattice(case, seed):
    """Full (both triangles) rows of the rescaled Hamiltonian and of the velocity operator:
    n, (cols, vals) of H, (cols, vals) of V or None, arrays of shape (n, entries per row); and the
    half band width the Hamiltonian was divided by."""
    rng = np.random.default_rng(seed)
    lx, ly, lz = case["lx"], case["ly"], case["lz"]
    if case["lattice"] in ("square", "cubic"):
        n, t, W = lx * ly * lz, 1.0, 2.0 if case["lattice"] == "cubic" else 1.0
        g = np.arange(n)
        x, y, z = g % lx, (g // lx) % ly, g // (lx * ly)
        at = lambda a, b, c: a % lx + lx * (b % ly + ly * (c % lz))
        cols = [g, at(x + 1, y, z), at(x - 1, y, z), at(x, y + 1, z), at(x, y - 1, z)]
        if case["lattice"] == "cubic":
            cols += [at(x, y, z + 1), at(x, y, z - 1)]
        half = 1.05 * (t * (len(cols) - 1) + W / 2)
        vals = np.full((n, len(cols)), t / half, np.complex128)
        vals[:, 0] = W * (rng.random(n) - 0.5) / half
        return n, (np.stack(cols, 1), vals), None, half
    spin = case["lattice"] == "kane_mele"
    t, W, so, rashba = (1.0, 0.5, 0.06, 0.05) if spin else (-2.7, 1.0, 0.0, 0.0)
    d = np.array([[1.0, 0.0], [-0.5, math.sqrt(3) / 2], [-0.5, -math.sqrt(3) / 2]]) * (1.0 if spin else 1.42)
    sites = 2 * lx * ly
    i, j = (v.ravel() for v in np.meshgrid(np.arange(lx), np.arange(ly), indexing="ij"))
    cell = lambda a, b: (a % lx) + lx * (b % ly)
    order = np.argsort(cell(i, j))
    i, j = i[order], j[order]  # cell (i, j) at place i + lx j
    eps = W * (rng.random(sites) - 0.5)
    half = 1.05 * (3 * abs(t) + 6 * so + 3 * 2 * rashba + W / 2)
    shifts = [(0, 0), (-1, 0), (0, -1)]  # cell of the B neighbour of A along d[k]
    a1, a2 = d[0] - d[1], d[0] - d[2]
    second = [((1, 0), a1, 1), ((-1, 0), -a1, -1), ((0, 1), a2, -1), ((0, -1), -a2, 1), ((-1, 1), a2 - a1, 1),
              ((1, -1), a1 - a2, -1)]
    orb = 2 if spin else 1
    n = sites * orb
    hc = np.zeros((sites, orb, 1 + 3 * orb + (6 if spin else 0)), np.int64)
    hv = np.zeros(hc.shape, np.complex128)
    nv = 3 + (4 if spin else 0)
    vc, vv = np.zeros((sites, orb, nv), np.int64), np.zeros((sites, orb, nv), np.complex128)
    for sub in (0, 1):
        rows = 2 * cell(i, j) + sub
        sign = 1 if sub == 0 else -1
        for s in range(orb):
            sz = (1, -1)[s] if spin else 1
            hc[rows, s, 0], hv[rows, s, 0] = orb * rows + s, eps[rows]
            e, w = 1, 0
            for k in range(3):
                nb = 2 * cell(i + sign * shifts[k][0], j + sign * shifts[k][1]) + 1 - sub
                dv = sign * d[k]
                u = dv / np.linalg.norm(dv)
                for s2 in range(orb):
                    h = t if s2 == s else 1j * rashba * (u[1] + (1j if s == 0 else -1j) * u[0])
                    hc[rows, s, e], hv[rows, s, e] = orb * nb + s2, h
                    e += 1
                    if s2 == s:  # i (x_row - x_col) H, times the spin for the spin current
                        vc[rows, s, w], vv[rows, s, w] = orb * nb + s2, -1j * dv[0] * h * sz
                        w += 1
            for (di, dj), v, nu in second if spin else []:
                nb = 2 * cell(i + di, j + dj) + sub
                h = 1j * so * nu * sign * sz
                hc[rows, s, e], hv[rows, s, e] = orb * nb + s, h
                e += 1
                if abs(v[0]) > 1e-12:
                    vc[rows, s, w], vv[rows, s, w] = orb * nb + s, -1j * v[0] * h * sz
                    w += 1
    flat = lambda c, v: (c.reshape(n, -1), v.reshape(n, -1))
    hc, hv = flat(hc, hv)
    return n, (hc, hv / half), flat(vc, vv), half


def _operator(n, rows):
    """The operator of full rows (the interface reads their upper triangle)."""
    cols, vals = rows
    rowptr = np.arange(n + 1, dtype=np.int64) * cols.shape[1]
    return lq.Operator.from_csr(n, rowptr, cols.ravel(), vals.ravel())


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _states(n, R, seed):
    """R random-phase vectors, R x n."""
    gen = torch.Generator(device=_device()).manual_seed(seed)
    u = torch.rand((R, n), generator=gen, device=_device(), dtype=torch.float64)
    return torch.polar(torch.full_like(u, 1 / math.sqrt(n)), 2 * math.pi * u)


def _table(case, seed):
    """A Hermitian moment table with the decay that a disordered lattice's has."""
    M = case["M"]
    rng = np.random.default_rng(seed)
    a = rng.standard_normal((M, M)) + 1j * rng.standard_normal((M, M))
    m = np.arange(M)
    a *= np.exp(-np.abs(m[:, None] - m[None, :]) / 20.0) / (1.0 + m[:, None] + m[None, :])
    return (a + a.conj().T) / 2


def prepare(case, seed):
    kind, R, M = case["kind"], case["R"], case["M"]
    if kind == "post_bastin":
        return {"case": case, "mu": _table(case, seed)}
    dev = _device()
    st = {"case": case}
    if kind == "realisations":
        ops = []
        for r in range(case["seeds"]):
            n, h, _, _ = _lattice(case, [seed, r])
            ops.append(_operator(n, h))
        st.update(H=ops, mu=torch.zeros(case["seeds"] * M, dtype=torch.complex128, device=dev))
    else:
        n, h, v, half = _lattice(case, seed)
        st.update(H=_operator(n, h), half=half)
        needs_v = kind != "dos" or case["velocity"]
        st["V"] = _operator(n, v) if needs_v else None
        size = {"dos": M, "time": M * case.get("steps", 0)}.get(kind, M * M)
        st["mu"] = torch.zeros(size, dtype=torch.complex128, device=dev)
        if kind in ("kubo_bastin", "kubo_greenwood"):
            st["out"] = torch.zeros(3 * case["nump"], dtype=torch.float64, device=dev)
    st["states"] = _states(n, R, seed)
    st["opts"] = lq.make_opts(precision=lq.PREC_MIXED if case["mixed"] else lq.PREC_FP64,
                              realisations=1 if kind == "realisations" else 0)
    torch.cuda.synchronize()  # the solver works on a stream of its own
    return st


def run(state):
    c, o = state["case"], state.get("opts")
    kind, R, M = c["kind"], c["R"], c["M"]
    if kind == "post_bastin":
        E, sigma = lq.bastin_from_moments(state["mu"], c["sites"], 17.0, 0.0, 10.0, xbound=0.99)
        return {"E": E, "sigma": sigma}
    H, st, mu = state["H"], state["states"], state["mu"]
    if kind == "dos":
        lq.moments1d_dev(H, state["V"], st, R, M, mu, opts=o)
        return mu
    if kind == "realisations":
        lq.moments1d_realisations_dev(H, st, R, M, mu, opts=o)
        return mu.view(c["seeds"], M)
    V = state["V"]
    if kind == "time":
        lq.moments_td_dev(H, V, V, st, R, M, c["steps"], 1.0, 2 * state["half"], 0.0, mu, opts=o)
        return mu.view(M, c["steps"])
    if kind == "moments2d":
        lq.moments2d_dev(H, V, V, st, R, M, mu, opts=o)
        return mu.view(M, M)
    n, out = c["nump"], state["out"]
    if kind == "kubo_bastin":
        lq.kubo_bastin_dev(H, V, V, st, R, M, n, 2 * state["half"], 0.0, mu, out, opts=o)
        return {"mu": mu.view(M, M), "E": out[:n], "sigma": out[n : 2 * n], "integrand": out[2 * n :]}
    lq.kubo_fft_dev(H, V, V, st, R, M, n, lq.KUBO_GREENWOOD, 2 * state["half"], 0.0, out, opts=o)
    return {"E": out[:n], "sigma": out[n : 2 * n]}


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------
def work(case):
    kind, R, M = case["kind"], case["R"], case["M"]
    if kind == "post_bastin":
        div = 30 * M
        return {"bytes": 16 * M * M + 16 * div, "flops": 8 * div * M * M}
    cells = case["lx"] * case["ly"] * case["lz"]
    n = cells * {"square": 1, "cubic": 1, "honeycomb": 2, "kane_mele": 4}[case["lattice"]]
    nh = n * {"square": 5, "cubic": 7, "honeycomb": 4, "kane_mele": 13}[case["lattice"]]
    nv = n * {"honeycomb": 3, "kane_mele": 7}.get(case["lattice"], 0)
    op = lambda nnz: 20 * nnz + 4 * (n + 1)
    S = case.get("seeds", 1)
    inputs = S * op(nh) + 16 * n * R
    if kind == "dos" and case["velocity"]:
        return {"bytes": inputs + op(nv) + 16 * M, "flops": 8 * R * (nv + M * (nh + n))}
    if kind in ("dos", "realisations"):  # two moments from one product
        return {"bytes": inputs + 16 * M * S, "flops": 8 * R * ((M + 1) // 2) * (nh + 2 * n)}
    if kind == "time":
        terms = int(_terms(case))
        flops = 8 * R * case["steps"] * (nv + M * (nh + n) + 2 * terms * (nh + n))
        return {"bytes": inputs + op(nv) + 16 * M * case["steps"], "flops": flops}
    recursion = 8 * R * M * (2 * nh + nv)
    if kind == "kubo_greenwood":
        p = case["nump"]
        sites = min(8 * M * M, 4 * 5 * p * math.log2(p))
        return {"bytes": inputs + op(nv) + 24 * p, "flops": recursion + sites * n * R}
    out = 16 * M * M + (24 * case["nump"] if kind == "kubo_bastin" else 0)
    return {"bytes": inputs + op(nv) + out, "flops": recursion + 8 * M * M * n * R}


def _terms(case):
    """Terms of the evolution series of one time step (about the argument of its Bessel functions)."""
    half = {"honeycomb": 1.05 * 8.6, "kane_mele": 1.05 * 3.91}[case["lattice"]]
    return half / HBAR + 20


# ---------------------------------------------------------------------------------------------
# the same results in plain 64-bit torch
# ---------------------------------------------------------------------------------------------
class _Rows:
    def __init__(self, rows):
        cols, vals = rows
        self.cols = torch.from_numpy(np.ascontiguousarray(cols.T)).to(_device())
        self.vals = torch.from_numpy(np.ascontiguousarray(vals.T)).to(_device())

    def __call__(self, x):
        """The operator times a block of columns (n x R)."""
        y = self.vals[0][:, None] * x[self.cols[0]]
        for k in range(1, len(self.cols)):
            y += self.vals[k][:, None] * x[self.cols[k]]
        return y


def _chebyshev(H, x, M):
    prev, cur = None, x
    for m in range(M):
        yield cur
        if m + 1 < M:
            nxt = H(cur)
            if prev is not None:
                nxt = nxt.mul_(2).sub_(prev)
            prev, cur = cur, nxt


def _dos(H, V, states, M):
    x = states.T.contiguous()
    first = V(x) if V is not None else x
    mu = torch.stack([torch.vdot(x.reshape(-1), t.reshape(-1)) for t in _chebyshev(H, first, M)])
    mu *= 2 / states.shape[0]
    mu[0] /= 2
    return mu


def _blocks(H, V, states, M):
    x = states.T.contiguous()
    L = torch.stack([t.reshape(-1) for t in _chebyshev(H, V(x), M)])
    Rt = torch.stack([V(t).reshape(-1) for t in _chebyshev(H, x, M)])
    return L, Rt


def _moments2d(L, Rt, R):
    raw = L.conj() @ Rt.T
    mu = (raw + raw.conj().T) / 2 * (4 / R)
    mu[0] /= 2
    mu[:, 0] /= 2
    return mu


def _crescent(n):
    """Place of each ascending energy among the transform's frequencies."""
    y = np.empty(n, np.int64)
    h = n // 2
    y[n - 1] = n - 1
    y[0 : 2 * h : 2] = np.arange(h)
    y[1 : 2 * h : 2] = n - 1 - np.arange(h)
    return torch.from_numpy(y[::-1].copy()).to(_device())


def _site_sums(L, Rt, n, bastin):
    """Sums over sites of the products of the transforms (Bastin: p and w; Greenwood: p)."""
    M = L.shape[0]
    m = torch.arange(M, dtype=torch.float64, device=L.device)
    q = math.pi / (M + 1)
    g = ((M - m + 1) * torch.cos(q * m) + torch.sin(q * m) / math.tan(q)) / (M + 1)
    g = g * torch.where(m == 0, 1.0, 2.0)
    pf = torch.polar(g, math.pi * m / (2 * n))[:, None]
    low = (torch.arange(n, device=L.device) < n // 2)[:, None]
    p = torch.zeros(n, dtype=torch.float64, device=L.device)
    w = torch.zeros_like(p)
    chunk = max(1, (1 << 25) // n)
    tr = lambda u: torch.fft.ifft(pf * u, n=n, dim=0) * n
    side = lambda z: torch.where(low, z, z.conj())
    for a in range(0, L.shape[1], chunk):
        b, k = L[:, a : a + chunk], Rt[:, a : a + chunk]
        rb, ib, rk, ik = tr(b.real), tr(b.imag), tr(k.real), tr(k.imag)
        cb, ck = torch.complex(rb.real, -ib.real), torch.complex(rk.real, ik.real)
        if not bastin:
            p += (cb * ck).real.sum(1)
            continue
        gk, gb = side(rk) + 1j * side(ik), (side(rb) + 1j * side(ib)).conj()
        p += (cb * gk + gb * ck).real.sum(1)
        del rb, ib, rk, ik, gk, gb
        mb, mk = m[:, None] * b, m[:, None] * k
        dgb = (side(tr(mb.real)) + 1j * side(tr(mb.imag))).conj()
        dgk = side(tr(mk.real)) + 1j * side(tr(mk.imag))
        w += (dgb * ck - cb * dgk).imag.sum(1)
    return p, w


def _sigma(L, Rt, R, n, sites, half, bastin):
    p, w = _site_sums(L, Rt, n, bastin)
    x = torch.cos(math.pi * (2 * torch.arange(n, dtype=torch.float64, device=L.device) + 0.5) / n)
    omega = sites / half ** 2
    order = _crescent(n)
    E = x[order]
    if not bastin:
        return half * E, (2 * omega * (p / R) / (1 - x * x) / (2 * math.pi))[order], None
    v = (x * (p / R) - torch.sqrt(1 - x * x) * (w / R)) / (1 - x * x) ** 2 * (omega / math.pi)
    v = v[order]
    s = torch.zeros_like(v)
    s[:-1] = torch.cumsum(v[:-1] * (E[1:] - E[:-1]), 0)
    return half * E, s, v


def _evolve(H, x, dt, half):
    """exp(-i dt half H / hbar) x by Taylor series of short steps."""
    parts = max(1, math.ceil(dt * half / HBAR))
    z = -1j * dt * half / HBAR / parts
    for _ in range(parts):
        term = x
        for k in range(1, 30):
            term = H(term) * (z / k)
            x = x + term
    return x


def _post_bastin(case, seed):
    M, n, a = case["M"], case["sites"], 17.0 / 2
    q = math.pi / (M + 1)
    m = torch.arange(M, dtype=torch.float64, device=_device())
    g = ((M - m + 1) * torch.cos(q * m) + torch.sin(q * m) * math.cos(q) / math.sin(q)) * q / math.pi
    mu = torch.from_numpy(_table(case, seed)).to(_device()) * g[:, None] * g[None, :]
    div = 30 * M
    x = -0.99 + torch.arange(div, dtype=torch.float64, device=_device()) * (2 * 0.99) / (div - 1)
    f, th = torch.sqrt(1 - x * x)[:, None], torch.acos(x)[:, None] * m
    delta = torch.cos(th) / f / math.pi
    dg = -1j * torch.polar(torch.ones_like(th), -th) * (x[:, None] + 1j * m * f) / f ** 3
    kern = -2 * n / a ** 2 * (delta * (dg @ mu.T).imag).sum(1)
    E = x[:-1] * a
    return {"E": E.cpu(), "sigma": torch.cumsum(kern[:-1] * (x[1:] - x[:-1]), 0).cpu()}


def exact(case, seed):
    kind, R, M = case["kind"], case["R"], case["M"]
    if kind == "post_bastin":
        return _post_bastin(case, seed)
    if kind == "realisations":
        each = R // case["seeds"]
        rows = [_lattice(case, [seed, r]) for r in range(case["seeds"])]
        states = _states(rows[0][0], R, seed)
        return torch.stack([_dos(_Rows(l[1]), None, states[r * each : (r + 1) * each], M) for r, l in enumerate(rows)])
    n, h, v, half = _lattice(case, seed)
    states = _states(n, R, seed)
    H, V = _Rows(h), _Rows(v) if v is not None else None
    if kind == "dos":
        return _dos(H, V if case["velocity"] else None, states, M)
    if kind == "time":
        left, right = V(states.T.contiguous()), states.T.contiguous()
        mu = torch.zeros((M, case["steps"]), dtype=torch.complex128, device=_device())
        for s in range(case["steps"]):
            for k, t in enumerate(_chebyshev(H, V(right), M)):
                mu[k, s] = torch.vdot(left.reshape(-1), t.reshape(-1))
            left, right = _evolve(H, left, 1.0, half), _evolve(H, right, 1.0, half)
        mu *= 2 / R
        mu[0] /= 2
        return mu
    L, Rt = _blocks(H, V, states, M)
    if kind == "moments2d":
        return _moments2d(L, Rt, R)
    if kind == "kubo_bastin":
        mu = _moments2d(L, Rt, R)
        E, sigma, integrand = _sigma(L, Rt, R, case["nump"], n, half, True)
        return {"mu": mu, "E": E, "sigma": sigma, "integrand": integrand}
    E, sigma, _ = _sigma(L, Rt, R, case["nump"], n, half, False)
    return {"E": E, "sigma": sigma}
