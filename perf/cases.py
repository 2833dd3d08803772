"""The work that a user of this framework has it do, for timing and comparing builds.

Most cases advance a field (or an ensemble of fields) by a few RK3 time steps
between two outputs of the velocity, which is the whole of a DNS; the others
are the statistics that a run takes every few steps and the line solves that
a caller with its own device arrays asks for.  Sizes, shear and damping are
those of this repository's workloads, tests and default deck, and ragged ones
between them.

listed() gives the cases, draw() more of the same ranges, prepare() what a
program holds before the call, run() one pass, work() the bytes and
operations it cannot do without, tolerance() how far two correct
implementations may be apart, exact() the result in plain FP64 torch.
"""
from __future__ import annotations

import ctypes as ct
import math

import numpy as np
import torch

from homogenenousshearturbulence_b200 import hst

PI = math.pi
RK = ((120.0 / 32.0, 2.0, 0.0), (120.0 / 8.0, 50.0 / 8.0, 34.0 / 8.0), (120.0 / 20.0, 90.0 / 20.0, 50.0 / 20.0))
UNIT_BOX = dict(alfa0=1.0, beta0=1.0, ly=2.0 * PI)
BASE = dict(kind="steps", precision="fp64", exact_shift=False, members=1, ystretch=0.0, s2=0.0, damping="none",
            cfl=False, steps=4, re=2000.0, dt=0.001, k0=6.0, **UNIT_BOX)


def _case(**kw):
    return dict(BASE, **kw)


def listed():
    return [
        # the smallest field in use (96^2 x 64), the CFL number read after
        # every step as the driver's time loop does: launches and latency
        _case(name="steps_96x96x64", nx=31, ny=64, nz=32, re=1000.0, k0=4.0, cfl=True, steps=8),
        # the default deck of the input file: nx = 63, ny = 128, nz = 63 in
        # the box 3 x 2 x 1, CFL number every step
        _case(name="steps_default_deck", nx=63, ny=128, nz=63, alfa0=2.0 * PI / 3.0, beta0=2.0 * PI, ly=2.0,
              re=1000.0, k0=12.0, dt=0.0005, cfl=True, steps=6),
        # the medium drop-in field, 384^2 x 256, FP64 and mixed precision
        _case(name="steps_384x384x256", nx=127, ny=256, nz=128, k0=8.0, steps=6),
        _case(name="steps_384x384x256_mixed", nx=127, ny=256, nz=128, k0=8.0, precision="mixed", steps=6),
        # the large field, 768^2 x 512 with the exact shear shift, FP64 and
        # mixed precision: the headline of the benchmark
        _case(name="steps_768x768x512", nx=255, ny=512, nz=256, k0=16.0, re=5000.0, exact_shift=True, steps=4),
        _case(name="steps_768x768x512_mixed", nx=255, ny=512, nz=256, k0=16.0, re=5000.0, exact_shift=True,
              precision="mixed", steps=4),
        # the widest planes (1536^2), thinner in y than the full field so that
        # several contexts fit: oscillating spanwise shear, the hard
        # large-scale damping, exact shift, mixed precision
        _case(name="steps_1536x1536x128_mixed", nx=511, ny=128, nz=512, k0=24.0, re=10000.0, dt=0.0005,
              exact_shift=True, s2=0.5, damping="hard", precision="mixed", steps=4),
        # a stretched grid with ragged sizes (384 x 256 planes, 150 rows) and
        # the soft damping
        _case(name="steps_ragged_stretched", nx=100, ny=150, nz=75, ystretch=0.8, damping="soft", cfl=True, steps=4),
        # power-of-two transforms (512 x 256) on 200 rows, exact shift and
        # spanwise shear
        _case(name="steps_512x256x200", nx=169, ny=200, nz=85, exact_shift=True, s2=0.3, steps=4),
        # an ensemble: eight realisations of 192^2 x 128 advanced together
        _case(name="ensemble_8x192x192x128_mixed", nx=63, ny=128, nz=64, re=1500.0, dt=0.002, precision="mixed",
              members=8, steps=6),
        # the statistics and the column energies of a 384^2 x 256 field
        _case(name="stats_384x384x256", kind="stats", nx=127, ny=256, nz=128, k0=8.0, steps=1),
        # the three line solves of a substep (D2V, eta, dv/dy) on the caller's
        # own device arrays
        _case(name="solves_128x257x256", kind="solves", nx=127, ny=256, nz=128, k0=8.0, steps=1),
    ]


def _padded(nx, nz):
    """The dealiased nxd, nzd: at least 3/2 of the modes, a power of two times at most one factor three."""

    def fit(n):
        while True:
            j = n
            while j % 2 == 0:
                j //= 2
            if j in (1, 3):
                return n
            n += 1

    return fit(3 * (nx + 1) // 2), fit(3 * nz)


def _points(c):
    return c["members"] * (c["nx"] + 1) * (2 * c["nz"] + 1) * c["ny"]


def draw(rng):
    """One more case: sizes over the listed ranges (their logarithm), odd
    ones and any even number of rows among them."""

    def log_int(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    while True:
        c = _case(exact_shift=rng.random() < 0.5, s2=rng.choice([0.0, 0.0, 0.5]),
                  damping=rng.choice(["none", "none", "none", "hard", "soft"]), cfl=rng.random() < 0.5)
        c["kind"] = rng.choice(["steps"] * 8 + ["stats", "solves"])
        if c["kind"] == "steps" and rng.random() < 0.4:
            # mixed precision runs padded lengths 96 .. 1536 and rows in
            # multiples of 32
            c["precision"] = "mixed"
            px, pz = (rng.choice([96, 192, 384, 768, 1536]) for _ in range(2))
            c["nx"] = rng.randint(px // 4, px // 3 - 1)
            c["nz"] = rng.randint(pz // 6 + 1, pz // 3)
            c["ny"] = 32 * log_int(1, 16)
            if _padded(c["nx"], c["nz"]) != (px // 2, pz):
                continue
        else:
            c["nx"], c["nz"], c["ny"] = log_int(15, 511), log_int(15, 512), 2 * log_int(16, 256)
        if c["kind"] == "steps" and rng.random() < 0.2:
            c["members"] = rng.randint(2, 12)
        if rng.random() < 0.2:
            c["ystretch"] = 0.8
        if c["kind"] != "steps":
            c["precision"], c["steps"] = "fp64", 1
        c["k0"] = min(16.0, max(4.0, c["ny"] / 24.0))
        n = _points(c)
        if 2.0e4 <= n <= 2.0e7:
            return c


# ------------------------------------------------------------------ inputs ----
def _deck(c):
    d = dict(nx=c["nx"], ny=c["ny"], nz=c["nz"], alfa0=c["alfa0"], beta0=c["beta0"], ly=c["ly"],
             ystretch=c["ystretch"], re=c["re"], S=1.0, deltat=c["dt"], exact_shift=c["exact_shift"],
             precision=c["precision"])
    if c["s2"]:
        d.update(s2_amplitude=c["s2"], s2_period=10.0)
    if c["damping"] != "none":
        d.update(damp_kpar=2.0 * c["alfa0"], damp_kperp=2.0 * c["beta0"])
        d.update(dict(damp_hard=True) if c["damping"] == "hard" else dict(damp_rate=0.5, damp_edge=0.3))
    return d


def _grid(c):
    """y(-2:ny+1), periodic beyond the box."""
    ny, ly, a = c["ny"], c["ly"], c["ystretch"]

    def ymap(xi):
        if a <= 1.0e-10:
            return xi
        if xi <= 0.5:
            return 0.5 * math.tanh(2.0 * a * xi) / math.tanh(a)
        return 0.5 * (2.0 + math.tanh(2.0 * a * (xi - 1.0)) / math.tanh(a))

    return np.array([ly * ymap((i % ny) / ny) + ly * float((i - i % ny) // ny) for i in range(-2, ny + 2)])


def _field(c, seed, y):
    """A seeded divergence-free field of energy 0.1 with E(k) ~ k^4
    exp(-2 (k/k0)^2), as (3, nx+1, 2nz+1, ny+4) on the GPU: the curl of a
    random vector potential, its ix = 0 plane Hermitian."""
    nx, ny, nz, a0, b0, ly, k0 = (c[k] for k in ("nx", "ny", "nz", "alfa0", "beta0", "ly", "k0"))
    f8, dev = torch.float64, "cuda" if torch.cuda.is_available() else "cpu"
    kcut = 4.0 * k0
    bx, bz = min(nx, int(kcut / a0)), min(nz, int(kcut / b0))
    bm = min(ny // 3, int(kcut * ly / (2.0 * PI)))
    kx = a0 * torch.arange(bx + 1, device=dev, dtype=f8)[:, None, None]
    kz = b0 * torch.arange(-bz, bz + 1, device=dev, dtype=f8)[None, :, None]
    ky = 2.0 * PI / ly * torch.arange(-bm, bm + 1, device=dev, dtype=f8)[None, None, :]
    g = torch.Generator(device=dev).manual_seed(int(seed))
    r = torch.randn((3, 2, bx + 1, 2 * bz + 1, 2 * bm + 1), generator=g, device=dev, dtype=f8)
    r = r * torch.exp(-(kx * kx + ky * ky + kz * kz) / (k0 * k0))
    A = torch.complex(r[:, 0], r[:, 1])
    del r
    A[:, 0] = 0.5 * (A[:, 0] + torch.conj(torch.flip(A[:, 0], (1, 2))))
    A[:, 0, bz] = 0.0
    E = torch.exp(1j * (ky[0, 0][:, None] * torch.from_numpy(y).to(dev)[None, :]))
    V = torch.zeros((3, nx + 1, 2 * nz + 1, ny + 4), dtype=torch.complex128, device=dev)
    for k, u in enumerate((lambda: ky * A[2] - kz * A[1], lambda: kz * A[0] - kx * A[2], lambda: kx * A[1] - ky * A[0])):
        V[k, :bx + 1, nz - bz:nz + bz + 1] = (1j * u()) @ E
    dyl = torch.from_numpy(0.5 * (y[3:ny + 3] - y[1:ny + 1])).to(dev)
    e = 0.0
    for k in range(3):
        q = ((V[k, :, :, 2:ny + 2].real.square() + V[k, :, :, 2:ny + 2].imag.square()) * dyl).sum((1, 2))
        e += float(2.0 * q.sum() - q[0])
    V *= math.sqrt(0.1 / (0.5 * e / ly))
    return V


def _solve_shift(c):
    """The wrap displacement of the line-solve case and its lambda (the
    third substep's)."""
    return 0.37 * 2.0 * PI / c["alfa0"], 0.21 * 2.0 * PI / c["beta0"], RK[2][0] / c["dt"]


def _line_solve(c, der, src, dst, kind, stream):
    f = hst.lib().hst_gpu_line_solve_noalloc
    if not f.argtypes:
        d, i, vp = ct.c_double, ct.c_int, ct.c_void_p
        f.restype = i
        f.argtypes = [i, i, i, d, d, d, i, d, vp, vp, vp, d, d, vp, ct.c_char_p, i]
    sx, sz, lam = _solve_shift(c)
    msg = ct.create_string_buffer(256)
    rc = f(c["nx"], c["ny"], c["nz"], c["alfa0"], c["beta0"], c["re"], kind, lam, der.data_ptr(), src.data_ptr(),
           dst.data_ptr(), sx, sz, stream, msg, 256)
    if rc != 0:
        raise RuntimeError(f"line solve {kind}: {msg.value.decode()}")


def prepare(case, seed):
    c = dict(BASE, **case)
    y = _grid(c)
    if c["kind"] == "solves":
        # right-hand sides of the two implicit systems, and v with its ghost rows
        V = _field(c, seed, y)
        s = hst.Solver(dict(_deck(c), nx=1, nz=1))  # the derivative table of this grid
        der = torch.from_numpy(np.ascontiguousarray(s.der).ravel()).cuda()
        s.close()
        return dict(case=c, der=der, rhs2=V[1] * 1.0e4, rhs1=V[0] * 1.0e4, v=_with_ghosts_last(c, V[1], *_solve_shift(c)[:2]),
                    out=[torch.zeros_like(V[0]) for _ in range(3)])
    s = hst.Solver(_deck(c), members=c["members"])
    s.time = 0.0
    out = torch.empty((c["members"], 3) + s.shape, dtype=torch.complex128, pin_memory=True)
    for m in range(c["members"]):
        if c["members"] > 1:
            s.select(m)
        out[m].copy_(_field(c, seed + 1000 * m, y))
        for k in range(3):
            s.upload_ptr(k, out[m, k].data_ptr())
            s.fill_ghosts(k)
    return dict(case=c, solver=s, out=out)


# -------------------------------------------------------------------- run ----
def run(state):
    c = state["case"]
    if c["kind"] == "solves":
        stream = torch.cuda.current_stream().cuda_stream
        for kind, src, dst in ((hst.KIND_D2V, state["rhs2"], state["out"][0]), (hst.KIND_ETA, state["rhs1"], state["out"][1]),
                               (hst.KIND_DY, state["v"], state["out"][2])):
            _line_solve(c, state["der"], src, dst, kind, stream)
        ny = c["ny"]
        return [o[:, :, 2:ny + 2] for o in state["out"]]  # the rows the solve writes
    s = state["solver"]
    if c["kind"] == "stats":
        sums, exz = s.outstats_sums()
        return dict(sums=np.array(list(sums.values())), exz=exz)
    if c["cfl"]:
        for _ in range(c["steps"]):
            s.timestep()
    else:
        s.timesteps(c["steps"])
    out = state["out"]
    for m in range(c["members"]):
        if c["members"] > 1:
            s.select(m)
        for k in range(3):
            s.download_async_ptr(k, out[m, k].data_ptr())
    return dict(V=out, cfl=s.cfl) if c["cfl"] else dict(V=out)


# ------------------------------------------------------------ work, tolerance ----
def work(case):
    """Bytes: every substep reads and writes the velocity and the two carried
    terms (ten complex FP64 fields).  Operations: the real transforms of
    three velocities and six products in x and z, 5 N log2 N a complex line,
    and about 600 a point for the stencils, products and line solves."""
    c = dict(BASE, **case)
    n = _points(c)
    if c["kind"] == "solves":
        return {"bytes": 16.0 * 6 * n, "flops": 3 * 60.0 * n}
    if c["kind"] == "stats":
        return {"bytes": 16.0 * 3 * n, "flops": 3 * 60.0 * n}
    nxd, nzd = _padded(c["nx"], c["nz"])
    NX, M = 2 * nxd, c["members"]
    fx = 9 * 2.5 * NX * math.log2(NX) * nzd * c["ny"] * M
    fz = 9 * 5.0 * nzd * math.log2(nzd) * (c["nx"] + 1) * c["ny"] * M
    sub = 3 * c["steps"]
    return {"bytes": sub * 160.0 * n, "flops": sub * (fx + fz + 600.0 * n)}


def tolerance(case):
    """Measured against exact(): FP64 up to 1e-13 relative after twelve
    substeps, mixed precision up to 3.2e-8 in V and 1.1e-7 in the CFL number
    (the largest value of an FP32 transform).  A single mode may be off by
    more than the whole field is: the field's norm is in a few modes."""
    if dict(BASE, **case)["precision"] == "mixed":
        return {"rel": 5e-7, "max": 1e-4}
    return {"rel": 5e-13, "max": 1e-10}


# ------------------------------------------------------------------ exact ----
class _Ref:
    """One time-stepping reference in FP64 torch: fields are [rows, members,
    nx+1, 2nz+1] with the rows first, ghost rows added where a stencil needs
    them."""

    def __init__(self, c):
        self.c = c
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.y = _grid(c)
        ny = self.ny = c["ny"]
        self.der = _der_table(self.y, ny)
        self.al = c["alfa0"] * torch.arange(c["nx"] + 1, device=self.dev, dtype=torch.float64)[:, None]
        self.be = c["beta0"] * torch.arange(-c["nz"], c["nz"] + 1, device=self.dev, dtype=torch.float64)[None, :]
        self.kk = self.al ** 2 + self.be ** 2
        self.dyl = 0.5 * (self.y[3:ny + 3] - self.y[1:ny + 1])
        self.nxd, self.nzd = _padded(c["nx"], c["nz"])
        self.s2a, self.w = c["s2"], 2.0 * PI / 10.0

    def shifts(self, t):
        c = self.c
        lx, lz = 2.0 * PI / c["alfa0"], 2.0 * PI / c["beta0"]
        return math.fmod(t * c["ly"], lx), self.s2_integral(0.0, t) * c["ly"] % lz

    def s2_integral(self, a, b):
        return self.s2a / self.w * (math.cos(self.w * a) - math.cos(self.w * b)) if self.s2a else 0.0

    def phase(self, sx, sz):
        return torch.exp(-1j * (self.al * sx + self.be * sz))

    def ghosts(self, f, ph):
        return torch.cat([f[-2:] * ph.conj(), f, f[:2] * ph])

    def sten(self, n, g):
        """the five-point stencil n (D0, D1, D2, D4) of g (with ghost rows)"""
        w = torch.from_numpy(self.der[:, n]).to(self.dev)[:, :, None, None, None]
        o = w[:, 0] * g[:self.ny]
        for j in range(1, 5):
            o.addcmul_(w[:, j].to(o.dtype), g[j:j + self.ny])
        return o

    def solve(self, rhs, ph, poly):
        """the cyclic pentadiagonal systems with rows sum_k kk^k poly[k]:
        elimination of rows 0 .. ny-3 of every column at once, bordered by
        the last two unknowns; rhs a list of [ny, ...] right-hand sides"""
        n, kk = self.ny, self.kk
        B = torch.stack(rhs, 1)  # [ny, K, M, nxB, nzT]
        K = B.shape[1]
        X = torch.zeros((n, K + 2) + B.shape[2:], dtype=B.dtype, device=self.dev)
        X[:, :K] = B
        P = [torch.from_numpy(np.ascontiguousarray(p)).to(self.dev) for p in poly]

        def row(i):
            a = P[0][i][:, None, None] + torch.zeros_like(kk)
            if len(P) > 1:
                a = a + P[1][i][:, None, None] * kk
            if len(P) > 2:
                a = a + P[2][i][:, None, None] * (kk * kk)
            return a

        phc = ph.conj()
        # the border's columns: coefficients of x[n-2] (K) and x[n-1] (K+1), to the right-hand side
        r0, r1, rm, rl = row(0), row(1), row(n - 4), row(n - 3)
        X[0, K] = -r0[0] * phc
        X[0, K + 1] = -r0[1] * phc
        X[1, K + 1] = -r1[0] * phc
        X[n - 4, K] = -rm[4]
        X[n - 3, K] = -rl[3]
        X[n - 3, K + 1] = -rl[4]
        U1, U2 = [], []
        for i in range(n - 2):
            a = row(i)
            a1, a2, a3 = a[1], a[2], a[3]
            if i >= 2:
                a1 = a1 - a[0] * U1[i - 2]
                a2 = a2 - a[0] * U2[i - 2]
                X[i] -= a[0] * X[i - 2]
            if i >= 1:
                a2 = a2 - a1 * U1[i - 1]
                a3 = a3 - a1 * U2[i - 1]
                X[i] -= a1 * X[i - 1]
            rp = 1.0 / a2
            U1.append(a3 * rp)
            U2.append(a[4] * rp)
            X[i] *= rp
        X[n - 4] -= U1[n - 4] * X[n - 3]
        for i in range(n - 5, -1, -1):
            X[i] -= U1[i] * X[i + 1] + U2[i] * X[i + 2]
        # the last two rows
        p, q = row(n - 2), row(n - 1)

        def part(i, k):  # the border rows' contribution of interior solution column k
            if i == 0:
                return p[0] * X[n - 4, k] + p[1] * X[n - 3, k] + p[4] * ph * X[0, k]
            return q[0] * X[n - 3, k] + ph * (q[3] * X[0, k] + q[4] * X[1, k])

        A = [[p[2] + part(0, K), p[3] + part(0, K + 1)], [q[1] + part(1, K), q[2] + part(1, K + 1)]]
        det = A[0][0] * A[1][1] - A[0][1] * A[1][0]
        out = []
        for k in range(K):
            b0, b1 = X[n - 2, k] - part(0, k), X[n - 1, k] - part(1, k)
            c0, c1 = (b0 * A[1][1] - b1 * A[0][1]) / det, (b1 * A[0][0] - b0 * A[1][0]) / det
            s = X[:n - 2, k] + c0 * X[:n - 2, K] + c1 * X[:n - 2, K + 1]
            out.append(torch.cat([s, c0[None], c1[None]]))
        return out

    def polys(self, kind, lam):
        d0, _, d2, d4 = (self.der[:, n] for n in range(4))
        ni = 1.0 / self.c["re"]
        if kind == "d2v":
            return [lam * d2 - ni * d4, -lam * d0 + 2.0 * ni * d2, -ni * d0]
        if kind == "eta":
            return [lam * d0 - ni * d2, ni * d0]
        return [d0]

    def damping(self, t):
        c = self.c
        if c["damping"] == "none":
            return None
        th = math.atan2(self.s2a * math.sin(self.w * t) if self.s2a else 0.0, 1.0)
        kp, kq = self.al * math.cos(th) + self.be * math.sin(th), -self.al * math.sin(th) + self.be * math.cos(th)
        r = torch.sqrt((kp / (2.0 * c["alfa0"])) ** 2 + (kq / (2.0 * c["beta0"])) ** 2)
        if c["damping"] == "hard":
            g = (r < 1.0 - 1.0e-6).to(torch.float64)
        else:
            x = (1.0 - r) / 0.3
            g = torch.where(r <= 0.7, 0.5 * torch.ones_like(r), 0.5 * x * x * (3.0 - 2.0 * x))
            g = torch.where(r < 1.0 - 1.0e-6, g, torch.zeros_like(r))
        g[0, c["nz"]] = 0.0
        return g

    def products(self, V, ph, want_cfl):
        """the six product spectra on every row, ghost rows included, and the CFL number"""
        c, nz, NX, NZ = self.c, self.c["nz"], 2 * self.nxd, self.nzd
        G = [self.ghosts(v, ph) for v in V]
        rows, out, cfl = self.ny + 4, [[] for _ in range(6)], 0.0
        step = max(1, int(2.0e8 / (NX * NZ * c["members"])))
        for a in range(0, rows, step):
            P = []
            for g in G:
                z = torch.zeros(g[a:a + step].shape[:3] + (NZ,), dtype=g.dtype, device=self.dev)
                z[..., :nz + 1] = g[a:a + step, ..., nz:]
                z[..., NZ - nz:] = g[a:a + step, ..., :nz]
                z = torch.fft.ifft(z, dim=-1, norm="forward")
                P.append(torch.fft.irfft(z, n=NX, dim=-2, norm="forward"))
            if want_cfl:
                lo, hi = max(a, 2), min(a + step, self.ny + 2)
                if lo < hi:
                    d = torch.from_numpy(self.dyl[lo - 2:hi - 2]).to(self.dev)[:, None, None, None]
                    u, v, w = (p[lo - a:hi - a].abs() for p in P)
                    m = u / (PI / (c["alfa0"] * self.nxd)) + v / d + w / (2.0 * PI / (c["beta0"] * NZ))
                    cfl = max(cfl, float(m.max()))
            for k, (i, j) in enumerate(((0, 0), (1, 1), (2, 2), (0, 1), (1, 2), (0, 2))):
                s = torch.fft.rfft(P[i] * P[j] / (NX * NZ), dim=-2)[..., :c["nx"] + 1, :]
                s = torch.fft.fft(s, dim=-1)
                out[k].append(torch.cat([s[..., NZ - nz:], s[..., :nz + 1]], -1))
        return [torch.cat(o) for o in out], cfl

    def substep(self, V, O, ode, dt, t, want_cfl):
        c, al, be, kk, ny = self.c, self.al, self.be, self.kk, self.ny
        ni, lam = 1.0 / c["re"], ode[0] / dt
        h = 2.0 / ode[0] * dt
        pt, pn = self.phase(*self.shifts(t)), self.phase(*self.shifts(t + h))
        Q, cfl = self.products(V, pt, want_cfl)
        u, v, w = (self.ghosts(f, pt) for f in V)
        s2 = self.s2a * math.sin(self.w * t) if self.s2a else 0.0
        g = self.damping(t)
        gs = g if c["damping"] == "soft" else torch.zeros_like(kk)
        mean = (0, c["nz"])
        v0, v2, v4 = (self.sten(n, v) for n in (0, 2, 3))
        unk = v2 - kk * v0
        r2 = lam * unk + ni * (v4 - 2.0 * kk * v2 + kk * kk * v0) - ode[2] * O[1] - ode[1] * gs * unk
        o2 = -gs * unk
        del v2, v4, unk
        f = 1j * (be * u - al * w)
        f[(slice(None), slice(None)) + mean] = torch.complex(u[(slice(None), slice(None)) + mean].real,
                                                             w[(slice(None), slice(None)) + mean].real)
        f0, f2 = self.sten(0, f), self.sten(2, f)
        ex = 1j * (s2 * al - be) * v0 - gs * f0
        r1 = lam * f0 + ni * (f2 - kk * f0) - ode[2] * O[0] + ode[1] * ex
        o1 = ex
        del f, f0, f2, v0
        for k, q in enumerate(Q):
            Q[k] = None
            q0, q1, q2 = (self.sten(n, q) for n in range(3))
            ru = rw = None
            if k == 0:
                ru, e = -1j * al * q0, -(al ** 2) * q1
            elif k == 1:
                e = kk * q1
            elif k == 2:
                rw, e = -1j * be * q0, -(be ** 2) * q1
            elif k == 3:
                ru, e = -q1, 1j * al * (q2 + kk * q0)
            elif k == 4:
                rw, e = -q1, 1j * be * (q2 + kk * q0)
            else:
                ru, rw, e = -1j * be * q0, -1j * al * q0, -2.0 * al * be * q1
            r2 += ode[1] * e
            o2 = o2 + e
            z = torch.zeros_like(q0)
            ru, rw = z if ru is None else ru, z if rw is None else rw
            e = 1j * (be * ru - al * rw)
            e[(slice(None), slice(None)) + mean] = torch.complex(ru[(slice(None), slice(None)) + mean].real,
                                                                 rw[(slice(None), slice(None)) + mean].real)
            r1 += ode[1] * e
            o1 = o1 + e
            del q, q0, q1, q2, ru, rw, e, z
        fs = [r1, r2, o1, o2]
        if c["damping"] == "hard":
            fs = [torch.where(g > 0.0, torch.zeros_like(x), x) for x in fs]
        gx = al * h + be * self.s2_integral(t, t + h)
        yy = torch.from_numpy(self.y[2:ny + 2]).to(self.dev)[:, None, None, None]
        e = torch.exp(-1j * gx * yy)
        if c["exact_shift"]:
            fs = [self.sten(0, self.ghosts(x * e, pn)) for x in self.solve(fs, pt, self.polys("d0", lam))]
        else:
            fs = [x * e for x in fs]
        r1, r2, o1, o2 = fs
        del fs, e
        kk0 = self.kk
        self.kk = kk.clone()
        self.kk[mean] = 1.0  # the mean of v is zero: its singular system is not solved
        v, = self.solve([r2], pn, self.polys("d2v", lam))
        self.kk = kk0
        v[(slice(None), slice(None)) + mean] = 0.0
        eta, = self.solve([r1], pn, self.polys("eta", lam))
        dv, = self.solve([self.sten(1, self.ghosts(v, pn))], pn, self.polys("dy", lam))
        rk = 1.0 / torch.where(kk == 0.0, torch.ones_like(kk), kk)
        u, w = 1j * rk * (al * dv - be * eta), 1j * rk * (be * dv + al * eta)
        m = (slice(None), slice(None)) + mean
        u[m] = eta[m].real.to(u.dtype)
        w[m] = eta[m].imag.to(u.dtype)
        return [u, v, w], [o1, o2], t + h, cfl


def _der_table(y, ny):
    """der[iy, n, j], n = D0, D1, D2, D4: the compact five-point coefficients
    of every row from their moment conditions, eliminated in extended precision."""
    x = np.stack([y[j:j + ny] - y[2:ny + 2] for j in range(5)], 1).astype(np.longdouble)  # [ny, 5]

    def solve(M, b):
        M, b = M.copy(), b.copy()
        n = np.arange(ny)
        for i in range(5):
            p = i + np.abs(M[:, i:, i]).argmax(1)
            M[n, i], M[n, p] = M[n, p].copy(), M[n, i].copy()
            b[n, i], b[n, p] = b[n, p].copy(), b[n, i].copy()
            for r in range(i + 1, 5):
                f = M[:, r, i] / M[:, i, i]
                M[:, r] -= f[:, None] * M[:, i]
                b[:, r] -= f * b[:, i]
        s = np.zeros_like(b)
        for i in range(4, -1, -1):
            s[:, i] = (b[:, i] - (M[:, i, i + 1:] * s[:, i + 1:]).sum(1)) / M[:, i, i]
        return s

    one = np.zeros((ny, 5), np.longdouble)
    V = np.stack([x ** (4 - i) for i in range(5)], 1)  # [ny, i, j]
    t = one.copy()
    t[:, 0] = 24.0
    d4 = solve(V, t)
    M = np.stack([np.longdouble((5 - i) * (6 - i) * (7 - i) * (8 - i)) * x ** (4 - i) for i in range(5)], 1)
    d0 = solve(M, np.stack([(d4 * x ** (8 - i)).sum(1) for i in range(5)], 1))
    t = one.copy()
    for i in range(3):
        t[:, i] = (d0 * (4 - i) * (3 - i) * x ** (2 - i)).sum(1)
    d2 = solve(V, t)
    t = one.copy()
    for i in range(4):
        t[:, i] = (d0 * (4 - i) * x ** (3 - i)).sum(1)
    d1 = solve(V, t)
    return np.stack([d0, d1, d2, d4], 1).astype(np.float64)


def _with_ghosts_last(c, f, sx, sz):
    """f (nx+1, 2nz+1, ny+4) with its ghost rows filled for a wrap displacement"""
    R = _Ref(c)
    ph = R.phase(sx, sz)[:, :, None]
    i = f[:, :, 2:-2]
    return torch.cat([i[:, :, -2:] * ph.conj(), i, i[:, :, :2] * ph], -1).contiguous()


def exact(case, seed):
    c = dict(BASE, **case)
    R = _Ref(c)

    def rows_first(f):
        return f[:, :, :, 2:-2].permute(3, 0, 1, 2).contiguous()

    V = torch.stack([_field(c, seed + 1000 * m, R.y) for m in range(c["members"])], 1)  # [3, M, nxB, nzT, rows]
    if c["kind"] == "solves":
        sx, sz, lam = _solve_shift(c)
        ph = R.phase(sx, sz)
        rhs2, rhs1 = rows_first(V[1] * 1.0e4), rows_first(V[0] * 1.0e4)
        R.kk[0, c["nz"]] = 1.0
        d2v, = R.solve([rhs2], ph, R.polys("d2v", lam))
        d2v[:, :, 0, c["nz"]] = 0.0
        R.kk[0, c["nz"]] = 0.0
        eta, = R.solve([rhs1], ph, R.polys("eta", lam))
        dy, = R.solve([R.sten(1, R.ghosts(rows_first(V[1]), ph))], ph, R.polys("dy", lam))
        return [f[:, 0].permute(1, 2, 0).contiguous() for f in (d2v, eta, dy)]
    F = [rows_first(v) for v in V]
    del V
    if c["kind"] == "stats":
        ph = R.phase(0.0, 0.0)
        wt = torch.from_numpy(R.dyl).to(R.dev)[:, None, None, None] * torch.where(R.al == 0.0, 1.0, 2.0)
        ab = lambda a, b: float((wt * (a.real * b.real + a.imag * b.imag)).sum())  # noqa: E731
        u, v, w = F
        e2 = sum(f.real ** 2 + f.imag ** 2 for f in F)
        eps = float((wt * R.kk * e2).sum())
        for f in F:
            d, = R.solve([R.sten(1, R.ghosts(f, ph))], ph, R.polys("dy", 0.0))
            eps += ab(d, d)
        g = R.damping(0.0)
        hit = torch.zeros_like(R.kk) if g is None else (g > 0.0).to(torch.float64)
        ed = float((wt * e2 * hit).sum())
        pd = 2.0 * float((wt * e2 * g).sum()) if c["damping"] == "soft" else 0.0
        sums = [eps, ab(u, v), ab(u, u), ab(v, v), ab(w, w), ab(w, v), ab(u, w), 0.0, 0.0, 0.0, ab(u, u) + ab(v, v) + ab(w, w),
                0.0, eps, ed, pd, float(hit.sum())]
        return dict(sums=np.array(sums), exz=(wt * e2).sum((0, 1)))
    O = [torch.zeros_like(F[0]), torch.zeros_like(F[0])]
    t, cfl = 0.0, 0.0
    for _ in range(c["steps"]):
        for i in range(3):
            F, O, t, q = R.substep(F, O, RK[i], c["dt"], t, c["cfl"] and i == 2)
            cfl = q if i == 2 else cfl
    ph = R.phase(*R.shifts(t))
    V = torch.stack([R.ghosts(f, ph).permute(1, 2, 3, 0) for f in F], 1)
    return dict(V=V, cfl=cfl) if c["cfl"] else dict(V=V)
