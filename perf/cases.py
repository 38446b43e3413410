"""The work a user of this framework has it do, as cases that a timing harness runs.

A case is a dict of plain values: an operation ("op"), a lattice with its parameters, a sector and
the operation's own sizes.  The operations are the package's public entry points:

  apply     y = H x on device vectors (Sector.apply), complex128
  lanczos   the alpha/beta chain of one start vector (Sector.lanczos), complex128
  ftlm      one sector's ln Z and E on a temperature grid (Sector.ftlm), complex128
  bchain    the 32-chain complex64 Lanczos of a sector (Sector.batched_lanczos)
  bftlm     one sector's ln Z and E from complex64 chains (Sector.batched_ftlm)
  sweep     every sector and the T x mu grid (grand_canonical_sweep), complex128 or batched complex64
  grad      ln Z_GC(U, V, t', mu, beta) and its gradient (autograd.grand_canonical_logz)
  kapply    y = H_K x in one momentum block (OrbitKBlock.apply), complex128
  kbftlm    one momentum block's ln Z and E from complex64 chains (OrbitKBlock.batched_ftlm)

exact() restates every operation in torch at 64 bits: the hop-by-hop action of H on the strings of
the two spin species, Lanczos chains from the same random start vectors and a dense eigen-solve of
each tridiagonal matrix.
"""
import math

import numpy as np
import torch

import ftlm_extended_hubbard_b200 as F
from ftlm_extended_hubbard_b200 import autograd as AG

T_GRID = np.round(np.arange(1, 21) * 0.1, 10)        # temperatures 0.1 .. 2.0
MU_GRID = np.round(np.arange(49) * 0.25 - 4.0, 10)   # chemical potentials -4 .. 8
HOST_START, DEVICE_START = "reference", "philox"


def _case(name, op, Lx, Ly, nu=0, nd=0, tp=-0.25, U=8.0, V=1.0, phi_x=0.0, phi_y=0.0, **more):
    c = {"op": op, "Lx": Lx, "Ly": Ly, "tp": tp, "U": U, "V": V, "phi_x": phi_x, "phi_y": phi_y, "nu": nu, "nd": nd}
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # One H v of the smallest lattice that the sweeps start from: a call that is all latency.
        _case("apply 4x2 (4,4)", "apply", 4, 2, 4, 4),
        # H v on a ragged mid-size sector with Peierls phases in both directions (no real hops on the wraps).
        _case("apply 4x3 (5,6)", "apply", 4, 3, 5, 6, phi_x=0.1, phi_y=0.2),
        # H v of the half-filled 4x4 lattice, the largest sector: the headline of the benchmark.
        _case("apply 4x4 (8,8)", "apply", 4, 4, 8, 8, phi_x=0.1),
        # The first steps of a spectrum run on a large sector.
        _case("lanczos 4x4 (6,6)", "lanczos", 4, 4, 6, 6, phi_x=0.1, M=10, start=DEVICE_START),
        # One sector of a finite-temperature study: a handful of chains, a temperature grid.
        _case("ftlm 4x3 (4,5)", "ftlm", 4, 3, 4, 5, R=4, M=60, start=DEVICE_START),
        # The whole grand-canonical study of a small lattice with the reference's start vectors.
        _case("sweep 4x2", "sweep", 4, 2, R=20, M=60, method="plain", start=HOST_START),
        # The same in complex64 blocks, on the lattice whose sectors are all of odd size.
        _case("sweep 3x3 batched", "sweep", 3, 3, R=32, M=60, method="batched", start=DEVICE_START),
        # The largest sector of the 4x3 lattice, 32 chains at once, as the batched sweeps run it.
        _case("bftlm 4x3 (6,6)", "bftlm", 4, 3, 6, 6, R=32, M=80),
        # The first block steps of a large 4x4 sector: what the big sweeps spend their hours on.
        _case("bchain 4x4 (5,6)", "bchain", 4, 4, 5, 6, phi_x=0.1, R=32, M=4),
        # Value and gradient of ln Z_GC with respect to the model's parameters (a fit's inner call).
        _case("grad 3x2", "grad", 3, 2, tp=-0.2, U=4.0, R=32, M=40, mu=2.0, beta=5.0),
        # H_K v in one momentum block.
        _case("kapply 4x4 (6,6)", "kapply", 4, 4, 6, 6, U=6.0, V=0.5, kx=1, ky=2),
        # 24 chains of one momentum block, as a momentum-resolved study runs each of its blocks.
        _case("kbftlm 4x4 (4,4)", "kbftlm", 4, 4, 4, 4, U=6.0, V=0.5, kx=1, ky=2, R=24, M=30),
    ]


def _log_between(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _sector(rng, lattices, lo, hi):
    """A sector of one of the lattices whose dimension is near a size drawn between lo and hi (by logarithm)."""
    Lx, Ly = rng.choice(lattices)
    n = Lx * Ly
    want = _log_between(rng, lo, hi)
    near = sorted((abs(math.log(math.comb(n, a) * math.comb(n, b) / want)), a, b)
                  for a in range(n + 1) for b in range(n + 1) if math.comb(n, a) * math.comb(n, b) <= hi)
    _, a, b = rng.choice(near[:6])
    return Lx, Ly, a, b


def draw(rng):
    tp = rng.choice([-0.25, -0.2, 0.3, round(rng.uniform(-0.5, 0.5), 3)])
    U, V = round(rng.uniform(1.0, 10.0), 2), round(rng.uniform(0.0, 2.0), 2)
    phi_x, phi_y = rng.choice([(0.0, 0.0), (0.1, 0.0), (0.0, 0.3), (0.1, 0.2)])
    par = dict(tp=tp, U=U, V=V, phi_x=phi_x, phi_y=phi_y)
    op = rng.choice(["apply", "apply", "lanczos", "ftlm", "sweep", "bftlm", "bchain", "grad", "kapply", "kbftlm"])
    start = rng.choice([HOST_START, DEVICE_START])
    if op == "apply":
        return _case("", op, *_sector(rng, [(4, 2), (3, 3), (4, 3), (3, 4), (5, 3), (4, 4)], 500, 2e8), **par)
    if op == "lanczos":
        return _case("", op, *_sector(rng, [(3, 3), (4, 3), (5, 3), (4, 4)], 2000, 7e7), **par, M=rng.randint(4, 10),
                     start=DEVICE_START)
    if op == "ftlm":
        return _case("", op, *_sector(rng, [(4, 2), (3, 3), (5, 2), (4, 3)], 500, 4e5), **par, R=rng.randint(2, 6),
                     M=rng.randint(30, 60), start=start)
    if op == "bftlm":
        return _case("", op, *_sector(rng, [(3, 3), (5, 2), (4, 3)], 1000, 9e5), **par, R=32, M=rng.randint(40, 80))
    if op == "bchain":
        return _case("", op, *_sector(rng, [(4, 3), (5, 3), (4, 4)], 2e4, 4e7), **par, R=32, M=rng.randint(2, 4))
    if op in ("kapply", "kbftlm"):
        lo, hi, lat = (5e3, 7e7, [(4, 3), (5, 3), (4, 4)]) if op == "kapply" else (4e3, 4e6, [(4, 3), (4, 4)])
        Lx, Ly, a, b = _sector(rng, lat, lo, hi)
        more = dict(kx=rng.randrange(Lx), ky=rng.randrange(Ly))
        if op == "kbftlm":
            more.update(R=rng.choice([8, 24, 32]), M=rng.randint(20, 30))
        return _case("", op, Lx, Ly, a, b, tp=tp, U=U, V=V, **more)
    Lx, Ly = rng.choice([(2, 2), (3, 2), (4, 2)])
    if op == "grad":
        return _case("", op, *rng.choice([(2, 2), (3, 2)]), **par, R=rng.choice([8, 32]), M=rng.randint(30, 40),
                     mu=round(rng.uniform(0.0, 4.0), 2), beta=round(rng.uniform(1.0, 5.0), 2))
    return _case("", op, Lx, Ly, **par, R=rng.randint(8, 20), M=rng.randint(40, 60),
                 method=rng.choice(["plain", "batched"]), start=start)


def _params(case):
    return F.HubbardParams(case["Lx"], case["Ly"], 1.0, case["tp"], case["U"], case["V"], case["phi_x"], case["phi_y"])


def _vector(dim, seed):
    """A normalised complex Gaussian vector, as the Lanczos runs hand to H."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = torch.randn(dim, 2, dtype=torch.float64, device="cuda", generator=g)
    return torch.view_as_complex(x / torch.linalg.vector_norm(x))


def prepare(case, seed):
    op = case["op"]
    st = {"case": case, "seed": seed % (1 << 30), "betas": 1.0 / T_GRID}
    if op in ("apply", "lanczos", "ftlm", "bftlm", "bchain", "kapply", "kbftlm"):
        st["h"] = F.Sector(_params(case), case["nu"], case["nd"])
        dim = st["h"].dim()
        if op in ("kapply", "kbftlm"):
            st["k"] = st["h"].orbit_block(case["kx"], case["ky"])
            dim = st["k"].dim
        if op in ("apply", "kapply"):
            st["x"] = _vector(dim, st["seed"])
            st["y"] = torch.empty_like(st["x"])
    elif op == "sweep":
        st["p"] = _params(case)
    else:
        g = torch.Generator()
        g.manual_seed(st["seed"])
        d = 0.01 * (torch.rand(5, dtype=torch.float64, generator=g) - 0.5)  # a point of a fit near the case's
        st["theta"] = torch.tensor([case["U"], case["V"], case["tp"], case["mu"], case["beta"]], dtype=torch.float64) + d
        st["lat"] = AG.Lattice(case["Lx"], case["Ly"], 1.0, case["phi_x"], case["phi_y"])
    return st


def run(st):
    c, seed = st["case"], st["seed"]
    op = c["op"]
    if op == "apply":
        st["h"].apply(st["x"], st["y"])
        return st["y"]
    if op == "kapply":
        st["k"].apply(st["x"], st["y"])
        return st["y"]
    if op == "lanczos":
        return st["h"].lanczos(c["M"], seed, c["start"])
    if op == "ftlm":
        return st["h"].ftlm(st["betas"], c["R"], c["M"], seed, c["start"])
    if op == "bchain":
        return st["h"].batched_lanczos(c["R"], c["M"], seed)
    if op == "bftlm":
        return st["h"].batched_ftlm(st["betas"], c["R"], c["M"], seed)
    if op == "kbftlm":
        return st["k"].batched_ftlm(st["betas"], c["R"], c["M"], seed)
    if op == "sweep":
        r = F.grand_canonical_sweep(st["p"], c["R"], c["M"], seed, T_GRID, MU_GRID, start=c["start"], method=c["method"])
        return {"lnz_s": r.lnz_sector, "e_s": r.e_sector, "lnz": r.lnz_gc, "n": r.n_avg, "e": r.e_avg}
    theta = st["theta"].clone().requires_grad_(True)
    lnz = AG.grand_canonical_logz(theta, st["lat"], c["R"], c["M"], seed, "batched", DEVICE_START)
    lnz.backward()
    return {"lnz": lnz.detach(), "grad": theta.grad}


# ---- the work a pass cannot do without -----------------------------------------------------------
def _sector_sizes(case, nu, nd):
    """(dimension, directed hops that end in one state on average) of a sector."""
    n = case["Lx"] * case["Ly"]
    links = len(_bonds(case))
    hops = sum(links * k * (n - k) / (n * (n - 1)) for k in (nu, nd)) if n > 1 else 0.0
    return math.comb(n, nu) * math.comb(n, nd), hops


def work(case):
    op, n = case["op"], case["Lx"] * case["Ly"]

    def chain(dim, hops, R, M, size):  # M steps: H v (one read, one write) and the update (three reads, one write)
        return R * M * dim * size * 6.0, R * M * dim * (8.0 * hops + 24.0)

    dim, hops = _sector_sizes(case, case["nu"], case["nd"])
    G = n if op in ("kapply", "kbftlm") else 1
    if op in ("apply", "kapply"):
        return {"bytes": 32.0 * dim / G, "flops": (8.0 * hops + 4.0) * dim / G}
    if op in ("lanczos", "ftlm"):
        b, f = chain(dim, hops, case.get("R", 1), case["M"], 16)
    elif op in ("bchain", "bftlm", "kbftlm"):
        b, f = chain(dim / G, hops, case["R"], case["M"], 8)
    else:
        b = f = 0.0
        for nu in range(n + 1):
            for nd in range(n + 1):
                d, h = _sector_sizes(case, nu, nd)
                if op == "grad":  # the chain, its replay and the operators' images of each vector
                    x, y = chain(d, h, case["R"], case["M"], 8)
                    b, f = b + 2.5 * x, f + 2.5 * y + 4.0 * case["R"] * d * case["M"] ** 2
                else:
                    x, y = chain(d, h, case["R"], case["M"], 16 if case["method"] == "plain" else 8)
                    b, f = b + x, f + y
    return {"bytes": b, "flops": f}


# ---- 64-bit restatement ---------------------------------------------------------------------------
def _bonds(case):
    """Directed hops {(from, to): coefficient}: c^dag_to c_from, duplicates summed."""
    Lx, Ly, out = case["Lx"], case["Ly"], {}

    def bond(x, y, dx, dy, t):
        X, Y = x + dx, y + dy
        wx, wy = (X >= Lx) - (X < 0), (Y >= Ly) - (Y < 0)
        i, j = y * Lx + x, (Y % Ly) * Lx + X % Lx
        if i == j or abs(t) < 1e-15:
            return
        ph = complex(math.cos(wx * case["phi_x"] + wy * case["phi_y"]), math.sin(wx * case["phi_x"] + wy * case["phi_y"]))
        out[i, j] = out.get((i, j), 0.0) - t * ph
        out[j, i] = out.get((j, i), 0.0) - t * ph.conjugate()

    for y in range(Ly):
        for x in range(Lx):
            if Lx > 1:
                bond(x, y, 1, 0, 1.0)
            if Ly > 1:
                bond(x, y, 0, 1, 1.0)
            for dx, dy in ((1, 1), (1, -1), (-1, 1), (-1, -1)):
                bond(x, y, dx, dy, case["tp"])
    return out


def _pairs(case):
    """Neighbour pairs of the V term, with multiplicity."""
    Lx, Ly, out = case["Lx"], case["Ly"], []
    for y in range(Ly):
        for x in range(Lx):
            for j, on in ((y * Lx + (x + 1) % Lx, Lx > 1), (((y + 1) % Ly) * Lx + x, Ly > 1)):
                if on and j != y * Lx + x:
                    out.append((y * Lx + x, j))
    return out


def _strings(n, k):
    """k-subsets of n sites in lexicographic order of their site lists, and mask -> rank."""
    import itertools
    m = np.array([sum(1 << s for s in c) for c in itertools.combinations(range(n), k)], dtype=np.int64)
    rank = np.full(1 << n, -1, dtype=np.int64)
    rank[m] = np.arange(m.size)
    return m, rank


def _odd(m):
    """Whether a mask has an odd number of sites."""
    m = np.array(m, dtype=np.int64)
    for s in (16, 8, 4, 2, 1):
        m = m ^ (m >> s)
    return m & 1


def _sign(bits):
    return torch.from_numpy(1.0 - 2.0 * bits.astype(np.float64)).cuda()


class _H:
    """H of one sector acting on tensors [Du, Dd, columns]."""

    def __init__(self, case, nu, nd, bonds=None, diag=True):
        n = self.n = case["Lx"] * case["Ly"]
        self.u, self.ru = _strings(n, nu)
        self.d, self.rd = _strings(n, nd)
        self.Du, self.Dd, self.dim = self.u.size, self.d.size, self.u.size * self.d.size
        occ_u = torch.from_numpy((self.u[:, None] >> np.arange(n)) & 1).double().cuda()
        occ_d = torch.from_numpy((self.d[:, None] >> np.arange(n)) & 1).double().cuda()
        adj = torch.zeros(n, n, dtype=torch.float64, device="cuda")
        for i, j in _pairs(case):
            adj[i, j] += 0.5
            adj[j, i] += 0.5
        self.docc = occ_u @ occ_d.T
        same = lambda o: ((o @ adj) * o).sum(1)  # noqa: E731
        self.pair = same(occ_u)[:, None] + same(occ_d)[None, :] + 2.0 * occ_u @ adj @ occ_d.T
        self.diag = (case["U"] * self.docc + case["V"] * self.pair)[:, :, None] if diag else None
        self.ups, self.dns = [], []
        for (f, t), c in sorted((_bonds(case) if bonds is None else bonds).items()):
            lo, hi = min(f, t), max(f, t)
            inner = sum(1 << s for s in range(lo + 1, hi))
            for own, rank, other, others, to in ((self.u, self.ru, self.d, sum(1 << s for s in range(lo, hi)), self.ups),
                                                 (self.d, self.rd, self.u, sum(1 << s for s in range(lo + 1, hi + 1)), self.dns)):
                out = np.nonzero(((own >> t) & 1 == 1) & ((own >> f) & 1 == 0))[0]
                if out.size:
                    src = own[out] ^ (1 << f) ^ (1 << t)
                    to.append((torch.from_numpy(out).cuda(), torch.from_numpy(rank[src]).cuda(), c, _sign(_odd(src & inner)),
                               _sign(_odd(other & others))))

    def __call__(self, x):
        y = self.diag * x if self.diag is not None else torch.zeros_like(x)
        for out, src, c, own, other in self.ups:
            y.index_add_(0, out, x.index_select(0, src) * (c * own[:, None, None] * other[None, :, None]))
        for out, src, c, own, other in self.dns:
            y.index_add_(1, out, x.index_select(1, src) * (c * other[:, None, None] * own[None, :, None]))
        return y

    def flat(self):
        """The same on [dim, columns]; a matrix product where H is small enough to be formed."""
        if self.dim <= 16000:
            eye = torch.eye(self.dim, dtype=torch.complex128, device="cuda")
            m = torch.cat([self(e.reshape(self.Du, self.Dd, -1)).reshape(self.dim, -1) for e in eye.split(1024, 1)], 1)
            return lambda v: m @ v
        return lambda v: self(v.reshape(self.Du, self.Dd, -1)).reshape(self.dim, -1)


def _philox(dim, key):
    """Complex Gaussians from Philox4x32-10 (counter: the element's index, key: (key, 0x7F4A7C15)) and Box-Muller."""
    i = torch.arange(dim, dtype=torch.int64, device="cuda")
    low = 0xFFFFFFFF
    c = [i & low, i >> 32, torch.zeros_like(i), torch.zeros_like(i)]
    k = [key & low, 0x7F4A7C15]
    for _ in range(10):
        a, b = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((b >> 32) & low) ^ c[1] ^ k[0], b & low, ((a >> 32) & low) ^ c[3] ^ k[1], a & low]
        k = [(k[0] + 0x9E3779B9) & low, (k[1] + 0xBB67AE85) & low]
    u1 = (((c[0] << 21) ^ (c[1] >> 11)) & ((1 << 53) - 1)).double().add_(0.5) * 2.0 ** -53
    u2 = (((c[2] << 21) ^ (c[3] >> 11)) & ((1 << 53) - 1)).double().add_(0.5) * 2.0 ** -53
    r = torch.sqrt(-2.0 * torch.log(u1))
    return torch.complex(r * torch.cos(2 * math.pi * u2), r * torch.sin(2 * math.pi * u2))


def _polar(dim, key):
    """Complex Gaussians from a 32-bit Mersenne twister and Marsaglia's polar method, the second of each pair first."""
    gen = np.random.MT19937()
    gen._legacy_seeding(key & 0xFFFFFFFF)
    got, have = [], 0
    while have < 2 * dim:
        raw = gen.random_raw(8 * dim + 64).astype(np.float64)
        v = 2.0 * ((raw[0::2] + raw[1::2] * 2.0 ** 32) * 2.0 ** -64) - 1.0
        x, y = v[0::2], v[1::2]
        r2 = x * x + y * y
        ok = (r2 <= 1.0) & (r2 > 0.0)
        x, y, r2 = x[ok], y[ok], r2[ok]
        m = np.sqrt(-2.0 * np.log(r2) / r2)
        got.append(np.stack([y * m, x * m], 1).reshape(-1))
        have += got[-1].size
    g = np.concatenate(got)[:2 * dim].reshape(dim, 2)
    return torch.view_as_complex(torch.from_numpy(np.ascontiguousarray(g))).cuda()


def _starts(dim, R, seed, start):
    v = torch.stack([(_philox if start == DEVICE_START else _polar)(dim, seed + r * 100003) for r in range(R)], 1)
    return v / torch.linalg.vector_norm(v, dim=0)


def _chains(h, v, M):
    """alpha [R, M], beta [R, M] (zero after a chain's end) and the steps used, by the plain recurrence."""
    R = v.shape[1]
    al, be = np.zeros((R, M)), np.zeros((R, M))
    used, alive = np.zeros(R, np.int32), np.ones(R, bool)
    q, prev, b = v, torch.zeros_like(v), torch.zeros(R, dtype=torch.float64, device=v.device)
    for k in range(M):
        w = h(q)
        z = (q.conj() * w).sum(0)
        w = w - z * q - b * prev
        n2 = (w.real ** 2 + w.imag ** 2).sum(0)
        a_k, n_k = z.real.cpu().numpy(), n2.cpu().numpy()
        al[alive, k] = a_k[alive]
        used[alive] = k + 1
        alive = alive & (n_k >= 1e-24)
        be[alive, k] = np.sqrt(n_k[alive])
        if not alive.any():
            break
        b = torch.sqrt(torch.clamp(n2, min=1e-30))
        prev, q = q, w / b
    return al, be, used


def _lnz(al, be, used, dim, betas):
    """ln Z and E of a sector from its chains: mean over chains of sum_k w_k exp(-beta l_k), times dim."""
    R, M = al.shape
    T = np.zeros((R, M, M))
    for k in range(M):
        T[:, k, k] = np.where(k < used, al[:, k], 1e6 + k)  # past a chain's end: decoupled, without weight
        if k + 1 < M:
            T[:, k, k + 1] = T[:, k + 1, k] = np.where(k + 1 < used, be[:, k], 0.0)
    lam, z = np.linalg.eigh(T)
    w = z[:, 0, :] ** 2
    on = (w > 0) & (lam < 5e5)
    x = np.where(on, np.log(np.where(on, w, 1.0)), -np.inf)[:, :, None] - np.where(on, lam, 0.0)[:, :, None] * betas
    top = x.max(axis=(0, 1))
    e = np.exp(x - top)
    s = e.sum(axis=(0, 1))
    return math.log(dim) + top + np.log(s / R), (e * np.where(on, lam, 0.0)[:, :, None]).sum(axis=(0, 1)) / s


def _grand(lnz_s, e_s, N, betas, mus, n):
    x = lnz_s[:, :, None] + betas[None, :, None] * mus[None, None, :] * N[:, None, None]
    top = x.max(0)
    w = np.exp(x - top)
    s = w.sum(0)
    return top + np.log(s), (w * N[:, None, None]).sum(0) / s / n, (w * e_s[:, :, None]).sum(0) / s


def _translations(case, h):
    """Per translation: its shift, image ranks, images and signs of the up and of the down strings, and per up string
    the down sites that it adds a sign with.  The fermionic modes are ordered by site, up before down on a site."""
    Lx, Ly, n, out = case["Lx"], case["Ly"], h.n, []
    for dy in range(Ly):
        for dx in range(Lx):
            to = [((s // Lx + dy) % Ly) * Lx + (s % Lx + dx) % Lx for s in range(n)]
            both = []
            for m, rank in ((h.u, h.ru), (h.d, h.rd)):
                img, odd = np.zeros_like(m), np.zeros_like(m)
                for a in range(n):
                    img |= ((m >> a) & 1) << to[a]
                    for b in range(a + 1, n):
                        if to[a] > to[b]:
                            odd ^= (m >> a) & (m >> b) & 1
                both.append((torch.from_numpy(rank[img]).cuda(), torch.from_numpy(img).cuda(), _sign(odd)))
            cross = np.zeros_like(h.u)
            for b in range(n):
                swaps = sum(1 << a for a in range(n) if (a <= b) != (to[a] <= to[b]))
                cross |= _odd(h.u & swaps) << b
            out.append((dx, dy, both[0], both[1], torch.from_numpy(cross).cuda()))
    return out


def _odd_of(m):
    """_odd() on a tensor of masks."""
    for s in (16, 8, 4, 2, 1):
        m = m ^ (m >> s)
    return (m & 1).double()


class _Block:
    """H_K on the momentum block's normalised orbit states, through the full space."""

    def __init__(self, case):
        self.h = h = _H(case, case["nu"], case["nd"])
        key = lambda u, d: ((u[:, None] << 16) | d[None, :]).reshape(-1)  # noqa: E731
        own = key(torch.from_numpy(h.u).cuda(), torch.from_numpy(h.d).cuda())
        moves = _translations(case, h)
        least = own
        for _, _, (_, iu, _), (_, idn, _), _ in moves:
            least = torch.minimum(least, key(iu, idn))
        reps = torch.nonzero(least == own).reshape(-1)
        reps = reps[torch.argsort(own[reps])]
        ru, rd = reps // h.Dd, reps % h.Dd
        A = torch.zeros(reps.numel(), dtype=torch.complex128, device="cuda")
        theta = lambda dx, dy: 2 * math.pi * (case["kx"] * dx / case["Lx"] + case["ky"] * dy / case["Ly"])  # noqa: E731
        downs = torch.from_numpy(h.d).cuda()
        eta = lambda su, sd, cross: su[ru] * sd[rd] * (1.0 - 2.0 * _odd_of(cross[ru] & downs[rd]))  # noqa: E731
        for dx, dy, (pu, _, su), (pd, _, sd), cross in moves:
            still = (pu[ru] == ru) & (pd[rd] == rd)
            t = theta(dx, dy)
            A += still * eta(su, sd, cross) * complex(math.cos(t), math.sin(t))
        keep = A.abs() > 1e-12
        self.reps, ru, rd = reps[keep], ru[keep], rd[keep]
        self.root = torch.sqrt(A.abs()[keep])
        self.dim = self.reps.numel()
        self.at = torch.full((h.dim,), self.dim, dtype=torch.int64, device="cuda")  # orbit of a state, none by default
        self.amp = torch.zeros(h.dim, dtype=torch.complex128, device="cuda")
        for dx, dy, (pu, _, su), (pd, _, sd), cross in moves:
            s = pu[ru] * h.Dd + pd[rd]
            t = theta(dx, dy)
            self.at[s] = torch.arange(self.dim, device="cuda")
            self.amp[s] = (eta(su, sd, cross) * self.root) * complex(math.cos(t), math.sin(t))

    def __call__(self, x):
        v = torch.cat([x, torch.zeros_like(x[:1])])
        f = self.amp[:, None] * v[self.at]
        y = self.h(f.reshape(self.h.Du, self.h.Dd, -1)).reshape(self.h.dim, -1)
        return y[self.reps] / self.root[:, None]


def _exact_sector(case, nu, nd, R, M, seed, start, betas):
    h = _H(case, nu, nd)
    if h.dim == 1:
        e = float(h.diag.item())
        return -betas * e, np.full(betas.size, e)
    al, be, used = _chains(h.flat(), _starts(h.dim, R, seed, start), M)
    return _lnz(al, be, used, h.dim, betas)


def _exact_grad(case, seed):
    """ln Z_GC and its derivatives from the full spectrum of every sector, on the chains' start vectors."""
    g = torch.Generator()
    g.manual_seed(seed)
    d = 0.01 * (torch.rand(5, dtype=torch.float64, generator=g) - 0.5)
    U, V, tp, mu, beta = (float(x) for x in torch.tensor([case["U"], case["V"], case["tp"], case["mu"], case["beta"]],
                                                         dtype=torch.float64) + d)
    c = dict(case, U=U, V=V, tp=tp)
    n = case["Lx"] * case["Ly"]
    only_tp = {k: v - _bonds(dict(c, tp=0.0)).get(k, 0.0) for k, v in _bonds(dict(c, tp=1.0)).items()}
    lz, en, N, dt = [], [], [], []
    for nu in range(n + 1):
        for nd in range(n + 1):
            h, hop = _H(c, nu, nd), _H(c, nu, nd, bonds=only_tp, diag=False)
            eye = torch.eye(h.dim, dtype=torch.complex128, device="cuda").reshape(h.Du, h.Dd, h.dim)
            lam, Z = torch.linalg.eigh(h(eye).reshape(h.dim, h.dim))
            v = _starts(h.dim, case["R"], seed, DEVICE_START) if h.dim > 1 else eye.reshape(1, 1)
            a = Z.conj().T @ v
            low = lam[0]
            w = torch.exp(-beta * (lam - low))
            p = (a.abs() ** 2).mean(1)
            q = (p * w).sum()
            lz.append(math.log(h.dim) + float(torch.log(q) - beta * low))
            en.append(float((p * w * lam).sum() / q))
            N.append(nu + nd)
            gap = lam[None, :] - lam[:, None]
            near = gap.abs() * beta < 1e-6
            mid = torch.exp(-beta * ((lam[None, :] + lam[:, None]) / 2 - low)) * beta
            K = torch.where(near, mid, (w[:, None] - w[None, :]) / torch.where(near, torch.ones_like(gap), gap))
            rho = (a @ a.conj().T) / a.shape[1] * K  # K_jk a_j a_k^*
            part = []
            for op in (lambda x: h.docc[:, :, None] * x, lambda x: h.pair[:, :, None] * x, hop):
                m = Z.conj().T @ op(eye).reshape(h.dim, h.dim) @ Z
                part.append(float(-(rho.T * m).sum().real / q))
            dt.append(part)
    lz, en, N, dt = (np.array(x) for x in (lz, en, N, dt))
    x = lz + beta * mu * N
    lnz = float(x.max() + np.log(np.exp(x - x.max()).sum()))
    w = np.exp(x - lnz)
    grad = [*(w[:, None] * dt).sum(0), beta * (w * N).sum(), (w * (mu * N - en)).sum()]
    return {"lnz": torch.tensor(lnz, dtype=torch.float64), "grad": torch.tensor(grad, dtype=torch.float64)}


def exact(case, seed):
    op, n = case["op"], case["Lx"] * case["Ly"]
    seed %= 1 << 30
    betas = 1.0 / T_GRID
    if op == "apply":
        h = _H(case, case["nu"], case["nd"])
        return h(_vector(h.dim, seed).reshape(h.Du, h.Dd, 1)).reshape(-1)
    if op == "kapply":
        b = _Block(case)
        return b(_vector(b.dim, seed)[:, None])[:, 0]
    if op == "lanczos":
        h = _H(case, case["nu"], case["nd"])
        al, be, used = _chains(h.flat(), _starts(h.dim, 1, seed, case["start"]), case["M"])
        k = int(used[0])
        nb = k if be[0, k - 1] > 0 else k - 1
        return al[0, :k], be[0, :nb], k
    if op == "ftlm":
        return _exact_sector(case, case["nu"], case["nd"], case["R"], case["M"], seed, case["start"], betas)
    if op == "bftlm":
        return _exact_sector(case, case["nu"], case["nd"], case["R"], case["M"], seed, DEVICE_START, betas)
    if op == "bchain":
        h = _H(case, case["nu"], case["nd"])
        f = h.flat()
        per = max(1, min(case["R"], int(2e8 // h.dim)))  # chains at once
        parts = [_chains(f, v, case["M"]) for v in _starts(h.dim, case["R"], seed, DEVICE_START).split(per, 1)]
        return tuple(np.concatenate(p) for p in zip(*parts))
    if op == "kbftlm":
        b = _Block(case)
        if b.dim <= 2 * case["M"]:  # the smallest blocks run other start vectors
            return None
        al, be, used = _chains(b, _starts(b.dim, case["R"], seed, DEVICE_START), case["M"])
        return _lnz(al, be, used, b.dim, betas)
    if op == "grad":
        return _exact_grad(case, seed)
    start = DEVICE_START if case["method"] == "batched" else case["start"]
    rows = [_exact_sector(case, nu, nd, case["R"], case["M"], seed, start, betas)
            for nu in range(n + 1) for nd in range(n + 1)]
    lz, es = np.stack([r[0] for r in rows]), np.stack([r[1] for r in rows])
    N = np.array([nu + nd for nu in range(n + 1) for nd in range(n + 1)], dtype=np.float64)
    gz, gn, ge = _grand(lz, es, N, betas, MU_GRID, n)
    return {"lnz_s": lz, "e_s": es, "lnz": gz, "n": gn, "e": ge}
