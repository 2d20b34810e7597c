"""The work that a user of this library has it do, as cases that can be timed and checked.

Three kinds of calls, all through the Python binding of the C ABI:

  solve     Context.solve: the lowest band frequencies at the points of a band path (the
            library's main call), in mixed precision or plain FP64;
  apply     Context.apply: one operator (Q_r, its adjoint, Q_r^* B^-1 Q_r, A_r^-1) on
            device vectors, what a caller with an eigensolver of its own runs;
  gradient  autograd.band_frequencies, forward and backward: one step of an inverse design.

The sizes are the repository's own: simple cubic grids from 16^3 to the benchmark's 96^3, the
FCC, BCC and hexagonal grids of the reference's lattices (Ny and Nz follow from Nx and the
lattice vectors, so they are odd or prime as often as not), and orthorhombic grids with three
different lengths.  The crystal is a pair of dielectric spheres of different size, placed
at random, and the k-points are a stretch of a path that leaves the Gamma point (where a case
says so) or lies off the symmetry planes, so no symmetry makes bands coincide.

exact() has its own restatement of the operators and a block Lanczos solver in plain torch, all in
64 bits.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fame-isotropic-gpu_b200"))
import fame_b200 as fb  # noqa: E402
from fame_b200.autograd import band_frequencies  # noqa: E402

OPS = {"qr": fb.OP_QR, "qrs": fb.OP_QRS, "qbq": fb.OP_QBQ, "invar": fb.OP_INVAR}
LATTICES = ("simple", "fcc", "bcc", "hex")

# per k-point of a solve: A_r^-1 applies, operator products in each, FP64 residuals in each
# (mixed precision) and restarts, as the 96^3 path's counters have them (10 bands, 40 steps)
APPLIES, PRODUCTS, RESIDUALS, RESTARTS = 82, 30, 2, 1.5


# ------------------------------------------------------------------ cases
def _solve(name, lattice, grid, nk, precision, tol, gamma=False, nwant=10, nstep=40):
    c = dict(kind="solve", lattice=lattice, nx=grid[0], ny=grid[1], nz=grid[2], nk=nk, precision=precision, tol=tol,
             gamma=gamma, nwant=nwant, nstep=nstep)
    return dict(c, name=name) if name else c


def _apply(name, lattice, grid, op, precision):
    c = dict(kind="apply", lattice=lattice, nx=grid[0], ny=grid[1], nz=grid[2], op=op, precision=precision)
    return dict(c, name=name) if name else c


def _gradient(name, lattice, grid, nwant):
    c = dict(kind="gradient", lattice=lattice, nx=grid[0], ny=grid[1], nz=grid[2], nwant=nwant)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one operator product on the smallest grid: a caller's own eigensolver while it is being
        # set up, all latency and launches
        _apply("product_16", "simple", (16, 16, 16), "qbq", "fp64"),
        # the same at the benchmark's grid, in the precision of the inner CG
        _apply("product_96_fp32", "simple", (96, 96, 96), "qbq", "fp32"),
        # a field projected back to the reduced space on a ragged general lattice
        _apply("project_fcc64", "fcc", (64, 55, 52), "qrs", "fp64"),
        # one A_r^-1 product (a whole CG solve) on a grid without a compile-time plan
        _apply("inverse_hex36", "hex", (36, 30, 26), "invar", "fp64"),
        # a short band path at the coarse resolution of a first look at a structure, from Gamma on
        _solve("path_32", "simple", (32, 32, 32), 12, "mixed", 1e-10, gamma=True),
        # a box with three different lengths, none a power of two
        _solve("path_box", "simple", (45, 66, 50), 4, "mixed", 1e-10, gamma=True),
        # the benchmark's grid and tolerance, in mixed precision (the largest case) and in FP64
        _solve("path_96", "simple", (96, 96, 96), 8, "mixed", 1e-12, gamma=True),
        _solve("point_96_fp64", "simple", (96, 96, 96), 1, "fp64", 1e-12),
        # the reference's other lattices at the resolution of its own runs
        _solve("path_fcc64", "fcc", (64, 55, 52), 8, "mixed", 1e-10, gamma=True),
        _solve("path_bcc48_fp64", "bcc", (48, 45, 39), 4, "fp64", 1e-10, nwant=12),
        _solve("point_hex128", "hex", (128, 107, 92), 1, "mixed", 1e-10, nwant=16),
        # one step of an inverse design on a voxel permittivity
        _gradient("design_32", "simple", (32, 32, 32), 8),
    ]


def draw(rng):
    """One more case: a grid of any of the lattices, the calls in about the same mix."""
    most = 0.1 * max(_cost(work(c)) for c in listed())
    while True:
        lattice = rng.choice(("simple", "simple", "fcc", "bcc", "hex"))
        n = int(round(math.exp(rng.uniform(math.log(12), math.log(100)))))
        if lattice == "simple":
            grid = (n, n, n) if rng.random() < 0.3 else tuple(max(8, int(round(n * rng.uniform(0.7, 1.3)))) for _ in range(3))
        else:
            grid = _grid_of(lattice, n)
        if not _fits(lattice, grid):
            continue
        kind = rng.choice(("solve", "solve", "solve", "apply", "apply", "gradient"))
        if kind == "apply":
            c = _apply(None, lattice, grid, rng.choice(("qr", "qrs", "qbq", "qbq", "invar")), rng.choice(("fp64", "fp32")))
            if c["op"] == "invar":
                c["precision"] = "fp64"
        elif kind == "gradient":
            c = _gradient(None, lattice, grid, rng.choice((4, 6, 8)))
        else:
            c = _solve(None, lattice, grid, rng.choice((1, 2, 3, 4, 6, 8, 12)), rng.choice(("mixed", "mixed", "fp64")),
                       rng.choice((1e-10, 1e-12)), rng.random() < 0.5, rng.choice((6, 8, 10, 12)), rng.choice((32, 40)))
        if _cost(work(c)) <= most:
            return c


def _fits(lattice, grid):
    """A plane has to fit the shared memory of one CTA in FP64.  Grids with a stage just under
    48 KB are left out too: the library refuses some of them."""
    fast, mid, slow = grid if lattice == "simple" else (grid[2], grid[1], grid[0])
    plane = mid * (fast | 1) + 2 * fast + 2 * mid
    stages = (8 * plane, 16 * plane, 392 * slow, 400 * slow)
    return plane <= 10400 and all(not 47000 < b <= 49152 for b in stages)


def _cost(w):
    return max(w["bytes"], w["flops"] / 8)


def work(case):
    """What a pass cannot do without.  A solve is taken at the iteration counts of the benchmark path."""
    N = case["nx"] * case["ny"] * case["nz"]
    fft = 3 * 5.0 * N * math.log2(N)  # one three-component transform

    def product(size):  # x in, y out, 1/eps in, and the field once out and once in
        return (4 * N + 6 * N) * 2 * size + 3 * N * size, 2 * fft + 120.0 * N

    if case["kind"] == "apply":
        size = 8 if case["precision"] == "fp64" else 4
        if case["op"] == "qbq":
            return {"bytes": (4 * N * 2 + 3 * N) * size, "flops": product(size)[1]}
        if case["op"] == "invar":
            b, f = product(8)
            return {"bytes": PRODUCTS * (b + 7 * 2 * N * 16), "flops": PRODUCTS * (f + 40.0 * N)}
        return {"bytes": (2 * N + 3 * N) * 2 * size, "flops": fft + 60.0 * N}
    nk = case.get("nk", 1)
    mixed = case.get("precision") == "mixed"
    nwant, nstep = case["nwant"], case.get("nstep", 40)
    b, f = product(4 if mixed else 8)
    s = 8 if mixed else 16
    per = APPLIES * PRODUCTS * (b + 7 * 2 * N * s)
    flops = APPLIES * PRODUCTS * (f + 40.0 * N)
    if mixed:
        rb, rf = product(8)
        per += APPLIES * RESIDUALS * (rb + 3 * 2 * N * 16)
        flops += APPLIES * RESIDUALS * rf
    per += APPLIES * (2 * (0.6 * nstep) + 4) * 2 * N * 16  # reorthogonalisation
    flops += APPLIES * 2 * (0.6 * nstep) * 8 * 2 * N
    per += (RESTARTS + 1) * (nstep + nwant) * 2 * N * 16
    return {"bytes": nk * per, "flops": nk * flops}


# ------------------------------------------------------------------ lattices
def _vectors(lattice):
    """Lattice vectors a1, a2, a3 of the computational frame, and the boundary shift t1."""
    r2, r3, r6 = math.sqrt(2.0), math.sqrt(3.0), math.sqrt(6.0)
    if lattice == "fcc":
        return np.array([[1 / r2, 0, 0], [0.5 / r2, r6 / 4, 0], [0.5 / r2, r6 / 12, 1 / r3]]), np.zeros(3)
    if lattice == "bcc":
        a = np.array([[r3 / 2, 0, 0], [-r3 / 6, 2 / r6, 0], [-r3 / 6, -1 / r6, 1 / r2]])
        return a, a[0] + a[1]
    return np.array([[1.2, 0, 0], [0, 1.0, 0], [0, -0.5, r3 / 2]]), np.array([0.0, 1.0, 0.0])  # hexagonal


def _grid_of(lattice, n):
    a, _ = _vectors(lattice)
    h = a[0, 0] / n
    return n, max(2, int(round(a[1, 1] / h))), max(2, int(round(a[2, 2] / h)))


def _lattice(case):
    """(grid, mesh lengths, lattice vectors (3, 3), simple, m, t1) of a case."""
    g = (case["nx"], case["ny"], case["nz"])
    if case["lattice"] == "simple":
        a = np.diag([v / g[0] for v in g])
        return g, np.full(3, 1.0 / g[0]), a, True, (0, 0, 0, 0), np.zeros(3)
    a, t1 = _vectors(case["lattice"])
    h = np.array([a[i, i] / g[i] for i in range(3)])
    b1 = a[1, 0] + (a[0, 0] if a[1, 0] < 0 else 0.0)
    a3 = a[2] + t1
    m = (int(round(b1 / h[0])), int(round(a3[0] / h[0])), int(a3[1] / h[1] + 0.49), 0)
    return g, h, a, False, m, t1


def _voxel_eps(case, rng):
    """Permittivity of the crystal at the three edge points of every cell: 3N doubles on the host."""
    g, h, a, *_ = _lattice(case)
    spheres = [(rng.uniform(0, 1, 3), rng.uniform(0.2, 0.26), rng.uniform(11, 13)),
               (rng.uniform(0, 1, 3), rng.uniform(0.12, 0.18), rng.uniform(8, 11))]
    size = min(np.linalg.norm(v) for v in a)
    A = torch.from_numpy(a).cuda()
    images = torch.cartesian_prod(*[torch.arange(-1.0, 2.0, dtype=torch.float64, device="cuda")] * 3) @ A
    eps = torch.ones(3, g[2], g[1], g[0], dtype=torch.float64, device="cuda")
    for e in range(3):
        axes = [(torch.arange(g[d], dtype=torch.float64, device="cuda") + (0.5 if d == e else 0.0)) * h[d] for d in (2, 1, 0)]
        z, y, x = torch.meshgrid(*axes, indexing="ij")
        fr = torch.stack([x, y, z], -1) @ torch.linalg.inv(A)
        for centre, radius, value in spheres:
            d = fr - torch.from_numpy(centre).cuda()
            d = (d - torch.round(d)) @ A
            near = torch.full(d.shape[:3], math.inf, dtype=torch.float64, device="cuda")
            for image in images:
                near = torch.minimum(near, (d + image).square().sum(-1))
            eps[e][near < (radius * size) ** 2] = value
    return eps.reshape(-1).cpu().numpy()


def _kpoints(case, rng):
    """nk wave vectors on a straight stretch of a band path, in the library's convention."""
    _, _, a, *_ = _lattice(case)
    nk = case.get("nk", 1)
    end = rng.uniform(0.15, 0.45, 3) * rng.choice((-1.0, 1.0), 3)
    start = np.zeros(3) if case.get("gamma") else end + rng.uniform(0.1, 0.3, 3) * rng.choice((-1.0, 1.0), 3)
    t = np.linspace(0.0, 1.0, nk)[:, None] if nk > 1 else np.ones((1, 1))
    theta = start + t * (end - start)
    return np.linalg.solve(a, theta.T).T.copy()


def _inputs(case, seed):
    rng = np.random.default_rng([seed, case["nx"], case["ny"], case["nz"]])
    N = case["nx"] * case["ny"] * case["nz"]
    d = {"N": N, "k": _kpoints(case, rng)}
    if case["kind"] == "gradient":
        d["eps"] = rng.uniform(1.0, 13.0, N)
        d["weights"] = rng.uniform(0.5, 1.5, case["nwant"])
    else:
        d["B"] = _voxel_eps(case, rng)
    if case["kind"] == "apply":
        n = 3 * N if case["op"] == "qrs" else 2 * N
        gen = torch.Generator(device="cuda").manual_seed(seed)
        x = torch.randn(n, 2, dtype=torch.float64, device="cuda", generator=gen)
        d["x"] = torch.view_as_complex(x).to(torch.complex128 if case["precision"] == "fp64" else torch.complex64)
    return d


# ------------------------------------------------------------------ one pass
def prepare(case, seed):
    d = _inputs(case, seed)
    g, h, a, simple, m, t1 = _lattice(case)
    ctx = fb.Context(g, h, a.reshape(-1), simple, m, t1)
    s = {"case": case, "ctx": ctx, "k": d["k"]}
    if case["kind"] == "gradient":
        s["eps"] = torch.from_numpy(d["eps"]).cuda().requires_grad_(True)
        s["weights"] = torch.from_numpy(d["weights"]).cuda()
        return s
    ctx.set_eps(d["B"])
    if case["kind"] == "apply":
        s["x"] = d["x"]
        s["y"] = torch.empty(3 * d["N"] if case["op"] == "qr" else 2 * d["N"], dtype=d["x"].dtype, device="cuda")
        s["params"] = fb.solver_params(ls_tol=1e-11, ls_maxit=1000)
    else:
        s["params"] = fb.solver_params(nwant=case["nwant"], nstep=case["nstep"], es_maxit=100, es_tol=case["tol"],
                                       ls_maxit=1000, ls_tol=case["tol"],
                                       precision=fb.MIXED if case["precision"] == "mixed" else fb.FP64)
    return s


def run(state):
    case, ctx = state["case"], state["ctx"]
    if case["kind"] == "solve":
        return {"freq": list(ctx.solve(state["k"], state["params"])["freq"])}
    if case["kind"] == "apply":
        ctx.apply(OPS[case["op"]], state["k"][0], state["x"], state["y"],
                  fb.FP64 if case["precision"] == "fp64" else fb.MIXED, state["params"])
        return {"y": state["y"]}
    eps = state["eps"]
    eps.grad = None
    w = band_frequencies(ctx, eps, state["k"][0], nwant=case["nwant"])
    (w * state["weights"]).sum().backward()
    return {"freq": w.detach(), "grad": eps.grad}


# ------------------------------------------------------------------ the same in plain torch, 64 bits
class _Operators:
    """Q_r, Q_r^* and Q_r^* B^-1 Q_r of one k-point on batches of vectors (rows)."""

    def __init__(self, case, k):
        g, h, a, simple, m, t1 = _lattice(case)
        self.g, self.simple = g, simple
        nx, ny, nz = g
        self.N = nx * ny * nz
        self.gamma = float(np.linalg.norm(k)) < (1e-4 if simple else 1e-3)
        f = lambda v: torch.as_tensor(v, dtype=torch.float64, device="cuda")  # noqa: E731
        ix, iy, iz = (torch.arange(n, dtype=torch.float64, device="cuda") for n in g)
        turn = lambda v: torch.polar(torch.ones_like(v), 2 * math.pi * v)  # noqa: E731
        if simple:
            th = a @ k
            lam = [(turn((i + t) / n) - 1) / s for i, t, n, s in zip((ix, iy, iz), f(th), g, f(h))]
            shape = (nz, ny, nx)
            L = [lam[0][None, None, :].expand(shape), lam[1][None, :, None].expand(shape), lam[2][:, None, None].expand(shape)]
            self.D = (turn(th[2] * iz / nz)[:, None, None] * turn(th[1] * iy / ny)[None, :, None] * turn(th[0] * ix / nx)[None, None, :])
        else:
            m1, m2, m3, _ = m
            c1 = -m1 / nx if a[1, 0] > 0 else 1 - m1 / nx if a[1, 0] < 0 else 0.0
            a2 = c1 * a[0] + a[1]
            a3 = a[2] - m3 / ny * a2 - m2 / nx * a[0] + t1
            tx, ty, tz = (float(np.dot(k, v)) for v in (a[0], a2, a3))
            sy = (ty - m1 / nx * ix)[:, None]
            sz = tz - m3 / ny * iy[None, :] + (m1 * m3 / (nx * ny) - m2 / nx) * ix[:, None]
            shape = (nx, ny, nz)
            L = [((turn((ix + tx) / nx) - 1) / h[0])[:, None, None].expand(shape),
                 ((turn((iy[None, :] + sy) / ny) - 1) / h[1])[:, :, None].expand(shape),
                 (turn((iz[None, None, :] + sz[:, :, None]) / nz) - 1) / h[2]]
            self.Dx = turn(tx * ix / nx)[:, None, None]
            self.Dy = turn(sy * iy[None, :] / ny)[:, :, None]
            self.Dz = turn(sz[:, :, None] * iz[None, None, :] / nz)
        x, y, z = (v.reshape(-1)[1 if self.gamma else 0:] for v in L)
        sq = lambda v: (v.conj() * v).real  # noqa: E731
        lq = sq(x) + sq(y) + sq(z)
        if simple:
            t = [5 * z - y, x - 3 * z, 3 * y - 5 * x]
            q = [v.conj() for v in t]
            p = [t[2] * y.conj() - t[1] * z.conj(), t[0] * z.conj() - t[2] * x.conj(), t[1] * x.conj() - t[0] * y.conj()]
            n2 = sum(sq(v) for v in t)
        else:
            s = x + y + z
            q = [z.conj() - y.conj(), x.conj() - z.conj(), y.conj() - x.conj()]
            p = [lq - v * s.conj() for v in (x, y, z)]
            n2 = sum(sq(v) for v in q)
        self.P = [v / torch.sqrt(n2 * lq) for v in p] + [v / torch.sqrt(n2) for v in q]
        self.sigma = torch.sqrt(lq).repeat(2)
        self.n = lq.numel()

    def qr(self, x):
        nx, ny, nz = self.g
        v = torch.zeros(x.shape[0], 3, self.N, dtype=x.dtype, device=x.device)
        for c in range(3):
            v[:, c, self.N - self.n:] = self.P[c] * x[:, :self.n] + self.P[3 + c] * x[:, self.n:]
        if self.simple:
            v = torch.fft.ifftn(v.view(-1, 3, nz, ny, nx), dim=(2, 3, 4)) * self.D
        else:
            v = torch.fft.ifft(v.view(-1, 3, nx, ny, nz), dim=4) * self.Dz
            v = torch.fft.ifft(torch.fft.ifft(v, dim=3) * self.Dy, dim=2) * self.Dx
            v = v.permute(0, 1, 4, 3, 2)
        return v.reshape(x.shape[0], 3 * self.N)

    def qrs(self, v):
        nx, ny, nz = self.g
        v = v.view(-1, 3, nz, ny, nx)
        if self.simple:
            v = torch.fft.fftn(v * self.D.conj(), dim=(2, 3, 4))
        else:
            v = torch.fft.fft(v.permute(0, 1, 4, 3, 2) * self.Dx.conj(), dim=2)
            v = torch.fft.fft(torch.fft.fft(v * self.Dy.conj(), dim=3) * self.Dz.conj(), dim=4)
        v = v.reshape(v.shape[0], 3, self.N)[:, :, self.N - self.n:]
        return torch.cat([sum(self.P[j + c].conj() * v[:, c] for c in range(3)) for j in (0, 3)], 1)

    def qbq(self, x, ib):
        return self.qrs(self.qr(x) * ib)

    def solve(self, b, ib, tol):
        """(Q_r^* B^-1 Q_r)^-1 b by CG, all rows at once."""
        x, r = torch.zeros_like(b), b.clone()
        p = r.clone()
        rr = (r.conj() * r).real.sum(1)
        stop = tol * tol * rr
        for it in range(400):
            q = self.qbq(p, ib)
            al = rr / (p.conj() * q).real.sum(1).clamp_min(1e-300)
            x += al[:, None] * p
            r -= al[:, None] * q
            new = (r.conj() * r).real.sum(1)
            p = r + (new / rr.clamp_min(1e-300))[:, None] * p
            rr = new
            if it % 4 == 3 and bool((rr <= stop).all()):
                break
        return x

    def inverse(self, x, ib, tol=1e-14):
        return self.solve(x / self.sigma, ib, tol) / self.sigma


def _bands(ops, ib, nwant, block=5, steps=30):
    """The lowest nwant frequencies and the eigenvectors y of A_r, by block Lanczos on A_r^-1 with
    full orthogonalisation."""
    gen = torch.Generator(device="cuda").manual_seed(3)
    w = torch.view_as_complex(torch.randn(block, 2 * ops.n, 2, dtype=torch.float64, device="cuda", generator=gen))
    w = w / ops.sigma ** 2  # near the low end of the spectrum
    m = block * steps
    U = torch.empty(m, 2 * ops.n, dtype=torch.complex128, device="cuda")
    AU = torch.zeros(m, m, dtype=torch.complex128, device="cuda")
    for s in range(steps):
        have = U[:s * block]
        for _ in range(2):
            if s:
                w = w - (w @ have.conj().T) @ have
            w = torch.linalg.qr(w.T)[0].T.contiguous()
        U[s * block:(s + 1) * block] = w
        w = ops.inverse(w, ib, 1e-13)
        AU[:(s + 1) * block, s * block:(s + 1) * block] = U[:(s + 1) * block].conj() @ w.T
    H = torch.triu(AU, 0)
    H = H + torch.triu(AU, 1).conj().T
    H.diagonal().copy_(AU.diagonal().real)
    th, Z = torch.linalg.eigh(H)
    th, Z = th.flip(0)[:nwant], Z.flip(1)[:, :nwant]
    return 1.0 / torch.sqrt(th), Z.T @ U


def exact(case, seed):
    d = _inputs(case, seed)
    N = d["N"]
    if case["kind"] == "apply":
        ops = _Operators(case, d["k"][0])
        x = d["x"].to(torch.complex128)[None]
        ib = 1.0 / torch.from_numpy(d["B"]).cuda()
        f = {"qr": ops.qr, "qrs": ops.qrs, "qbq": lambda v: ops.qbq(v, ib), "invar": lambda v: ops.inverse(v, ib)}
        return {"y": f[case["op"]](x)[0]}
    if case["kind"] == "gradient":
        ops = _Operators(case, d["k"][0])
        e = torch.from_numpy(d["eps"]).cuda()
        w, y = _bands(ops, 1.0 / e.repeat(3), case["nwant"], steps=40)
        E = ops.qr(y * ops.sigma).view(-1, 3, N) / e
        a2 = (E.conj() * E).real.sum(1)
        g = -(torch.from_numpy(d["weights"]).cuda() * w / 2 / (a2 @ e)) @ a2
        return {"freq": w, "grad": g}
    nk = case["nk"]
    most = max(1, min(nk, int(6e5 / N)))  # k-points that a few seconds are enough for
    rows = []
    for i in range(nk):
        if i not in {nk - 1 - j * nk // most for j in range(most)}:
            rows.append(None)
            continue
        ops = _Operators(case, d["k"][i])
        gamma = ops.gamma
        w, _ = _bands(ops, 1.0 / torch.from_numpy(d["B"]).cuda(), case["nwant"] - (2 if gamma else 0))
        rows.append(torch.cat([torch.zeros(2, dtype=torch.float64, device="cuda"), w]) if gamma else w)
    return {"freq": rows}
