"""The forward map as programs use it: matvecs (direct and IFGF, FP64 and complex64, one vector and
many), GMRES solves (one obstacle, many obstacles, preconditioned), and the off-surface field.

listed() names the workloads, draw() gives others of the same ranges.  prepare() builds the
operator and the seeded inputs, run() is one pass through the public interface, exact() the
result from a spectrally accurate Nystrom method (Kress's logarithmic splitting on the uniform
parameter grid) in 64 bits with torch alone, and work() the bytes and operations of one pass.
"""
import math

import numpy as np
import torch

import ifgf2d_gb300 as G

KITE_PATCHES = 1.024      # patches per wavenumber unit of the kite workloads (16 nodes: 10 points per wavelength and more)
DELTA = 0.01              # near-singular distance of the listed workloads


def listed():
    return [
        # the smallest call: the unit circle at k = 10 with 200 unknowns, direct operator, vectors on the GPU
        dict(name="direct_n200", op="direct", curve="circle", k=10.0, patches=20, Np=10, form="combined"),
        # a small matvec through host vectors, as a LinearOperator under a host solver calls it
        dict(name="host_k100", op="host", curve="kite", k=100.0, patches=128, Np=16, form="combined"),
        # the headline matvec: kite k = 500, N = 8192, FP64, vectors on the GPU
        dict(name="apply_k500", op="apply", curve="kite", k=500.0, patches=512, Np=16, form="combined"),
        # the same at N = 32768, the operator of the many-angle workload
        dict(name="apply_k2000", op="apply", curve="kite", k=2000.0, patches=2048, Np=16, form="combined"),
        # the complex64 matvec inside the refinement solves, at the headline size
        dict(name="mixed_k500", op="mixed", curve="kite", k=500.0, patches=512, Np=16, form="combined"),
        # and at the largest problem, N = 131072
        dict(name="mixed_k8000", op="mixed", curve="kite", k=8000.0, patches=8192, Np=16, form="combined"),
        # 64 densities against one FP64 operator (the residual of batched refinement, response matrices)
        dict(name="batch_k500_r64", op="batch", curve="kite", k=500.0, patches=512, Np=16, form="combined", nrhs=64),
        # 64 incidence angles, complex64: the inner matvec of the batched solve
        dict(name="batch_mixed_k2000_r64", op="batch_mixed", curve="kite", k=2000.0, patches=2048, Np=16, form="combined", nrhs=64),
        # a whole program in the plain form: constructor, set-up and FP64 GMRES at the default tolerance
        dict(name="solve_k500", op="solve", curve="kite", k=500.0, patches=512, Np=16, form="combined"),
        # one more incidence on a prepared operator in the chosen form (spectral preconditioner, refinement)
        dict(name="solve_spectral_k2000", op="solve_spectral", curve="kite", k=2000.0, patches=2048, Np=16, form="combined"),
        # many obstacles as one operator: 12 stars of uneven size, lock-step preconditioned GMRES
        dict(name="group_solve_12", op="group", members=12, kmin=40.0, kmax=300.0, geometry=1, Np=16, form="combined"),
        # the scattered field of a density on scattered off-surface points
        dict(name="field_k500", op="field", curve="kite", k=500.0, patches=512, Np=16, form="combined", targets=16385),
    ]


def draw(rng):
    op = rng.choice(["direct", "host", "apply", "mixed", "batch", "batch_mixed", "solve", "solve_spectral", "group", "field"])

    def log(a, b):
        return math.exp(rng.uniform(math.log(a), math.log(b)))

    if op == "group":
        return dict(op=op, members=rng.randint(2, 12), kmin=40.0, kmax=round(log(80.0, 300.0), 1), geometry=rng.randint(2, 10 ** 6),
                    Np=16, form="combined")
    hi = dict(direct=500.0, host=500.0, apply=2000.0, mixed=8000.0, batch=500.0, batch_mixed=2000.0, solve=500.0,
              solve_spectral=2000.0, field=500.0)[op]
    k = round(log(10.0 if op == "direct" else 60.0, hi), 2)
    curve = "circle" if op == "direct" and rng.random() < 0.5 else "kite"
    patches = max(20, int(math.ceil(k * KITE_PATCHES)) + rng.randint(0, 7))
    if curve == "kite":
        patches = max(64, patches)
    solving = op in ("solve", "solve_spectral")
    # long patches take a near-singular distance of their own scale
    delta = max(DELTA, round(0.6 * (2 * math.pi if curve == "circle" else 9.4) / patches, 4))
    c = dict(delta=delta, op=op, curve=curve, k=k, patches=patches, Np=16 if solving else rng.choice([10, 16, 16]),
             form="combined" if solving else rng.choice(["combined", "combined", "single_layer"]))
    if op in ("batch", "batch_mixed"):
        c["nrhs"] = rng.choice([1, rng.randint(2, 64), 64])
    if op == "field":
        c["targets"] = int(log(100, 16000)) | 1
    return c


# ---------------------------------------------------------------- inputs
def _waves(case, seed, nrhs):
    """Densities as sums of plane waves of the operator's wavenumber (what the Krylov vectors of a
    scattering solve look like): amplitudes and directions from the seed, [nrhs][6]."""
    g = np.random.default_rng([int(seed), 7])
    amp = (g.standard_normal((nrhs, 6)) + 1j * g.standard_normal((nrhs, 6))) / math.sqrt(12.0)
    ang = g.uniform(0.0, 2 * np.pi, (nrhs, 6))
    return amp, ang


def _density(case, seed, x, y, nrhs=1):
    """[nrhs][len(x)] on x's device"""
    amp, ang = _waves(case, seed, nrhs)
    dev = x.device
    out = torch.zeros(nrhs, x.numel(), dtype=torch.complex128, device=dev)
    for r in range(nrhs):
        for a, t in zip(amp[r], ang[r]):
            ph = case["k"] * (math.cos(t) * x + math.sin(t) * y)
            out[r] += complex(a) * torch.complex(torch.cos(ph), torch.sin(ph))
    return out


def _angle(seed):
    return float(np.random.default_rng([int(seed), 11]).uniform(0.0, 2 * np.pi))


def _stars(case, seed):
    """the members' shapes and wavenumbers (from the case) and incidence angles (from the seed)"""
    g = np.random.default_rng([int(case["geometry"]), 13])
    s = np.random.default_rng([int(seed), 17])
    out = []
    for _ in range(case["members"]):
        a, b = g.uniform(-0.05, 0.05, 5), g.uniform(-0.05, 0.05, 5)
        k = float(g.uniform(case["kmin"], case["kmax"]))
        patches = max(16, int(math.ceil(10 * k * 2 * math.pi * 1.05 / (2 * math.pi) / 16)))
        out.append((a, b, k, patches, float(s.uniform(0.0, 2 * np.pi))))
    return out


def _targets(case, seed):
    """off-surface points: a ring of the plane around the obstacle, 1 < distance scale < 2.5"""
    g = np.random.default_rng([int(seed), 19])
    r = g.uniform(2.6, 5.0, case["targets"])
    t = g.uniform(0.0, 2 * np.pi, case["targets"])
    return r * np.cos(t), r * np.sin(t)


def _map(case):
    curve = G.Circle() if case["curve"] == "circle" else G.Kite()
    return G.ForwardMap(case.get("delta", DELTA), [curve], (), 1.0, case["k"], Np=case["Np"], patches_per_curve=case["patches"], formulation=case["form"])


def prepare(case, seed):
    op, dev = case["op"], "cuda"
    if op == "group":
        fms, rhs = [], []
        for a, b, k, patches, ang in _stars(case, seed):
            fm = G.ForwardMap(DELTA, [G.Star(a, b)], (), 1.0, k, Np=case["Np"], patches_per_curve=patches, formulation="combined")
            fm.prepare(k, 0)
            fms.append(fm)
            rhs.append(-np.exp(1j * k * (math.cos(ang) * fm.xs_ + math.sin(ang) * fm.ys_)))
        g = G.Group(fms)
        for fm in fms:
            fm.close()
        return dict(case=case, g=g, rhs=np.concatenate(rhs))
    if op == "solve":
        return dict(case=case, angle=_angle(seed))
    fm = _map(case)
    s = dict(case=case, fm=fm)
    x, y = torch.from_numpy(fm.xs_).to(dev), torch.from_numpy(fm.ys_).to(dev)
    if op in ("direct", "field"):
        fm.compute_precomputations(case["k"])
    else:
        fm.precomps_and_setup(case["k"], 0)
    if op in ("batch", "batch_mixed"):
        s["x"] = _density(case, seed, x, y, case["nrhs"])
        s["y"] = torch.empty_like(s["x"])
    elif op == "solve_spectral":
        fm.spectral_setup()
        a = _angle(seed)
        s["rhs"] = -np.exp(1j * case["k"] * (math.cos(a) * fm.xs_ + math.sin(a) * fm.ys_))
    elif op == "field":
        s["tx"], s["ty"] = _targets(case, seed)
        s["x"] = _density(case, seed, x, y)[0].cpu().numpy()
    elif op == "host":
        s["x"] = _density(case, seed, x, y)[0].cpu().numpy()
    else:
        s["x"] = _density(case, seed, x, y)[0].contiguous()
        s["y"] = torch.empty_like(s["x"])
    return s


def run(s):
    case = s["case"]
    op = case["op"]
    if op in ("direct", "apply", "mixed"):
        s["fm"].apply_device(s["x"], s["y"], accelerated=op != "direct", mixed=op == "mixed")
        return s["y"]
    if op in ("batch", "batch_mixed"):
        s["fm"].apply_batch_device(s["x"], s["y"], case["nrhs"], mixed=op == "batch_mixed")
        return s["y"]
    if op == "host":
        return s["fm"].compute_Ax_acc(s["x"])
    if op == "field":
        return s["fm"].propagate_unacc(s["tx"], s["ty"], s["x"])
    if op == "solve_spectral":
        return s["fm"].solve_flexible(s["rhs"], "spectral", mixed=True)
    if op == "group":
        return s["g"].solve(s["rhs"], tol=1e-10, mixed=True, precond="spectral")
    fm = _map(case)                                  # op == "solve": the whole program
    a, k = s["angle"], case["k"]
    x = fm.solve(-np.exp(1j * k * (math.cos(a) * fm.xs_ + math.sin(a) * fm.ys_)), k)
    fm.close()
    return x


# ---------------------------------------------------------------- work
def _unknowns(case):
    if case["op"] == "group":
        return sum(p * case["Np"] for _, _, _, p, _ in _stars(case, 0))
    return case["patches"] * case["Np"]


def work(case):
    """Vectors read and written once, and the singular-correction weights (Np complex values per
    point), which have no cheaper form.  Operations of the IFGF: leaf sums, interpolations and
    near field at 5 x 5 cones come to about 4100 flops per point and binary level of the tree; of
    the direct sums: 150 per pair (a Hankel pair of one argument and a complex multiply-add)."""
    N, op = _unknowns(case), case["op"]
    nrhs = case.get("nrhs", 1)
    ifgf = 4100.0 * N * math.log2(N)
    weights = 16.0 * N * case["Np"]
    if op == "direct":
        return dict(bytes=32.0 * N + weights, flops=150.0 * N * N)
    if op == "field":
        return dict(bytes=32.0 * case["targets"] + 16.0 * N, flops=150.0 * N * case["targets"])
    if op in ("host", "apply", "mixed", "batch", "batch_mixed"):
        return dict(bytes=32.0 * N * nrhs + weights, flops=ifgf * nrhs)
    its = 25 if op in ("solve_spectral", "group") else 40      # a solve: its iterations' matvecs
    return dict(bytes=its * (32.0 * N + weights), flops=its * ifgf)


# ---------------------------------------------------------------- 64-bit values without the package
def _curve(case, t, star=None):
    """x, y and their first and second derivatives in t"""
    c, s = torch.cos(t), torch.sin(t)
    if star is not None:
        a, b = star
        r, dr, ddr = torch.ones_like(t), torch.zeros_like(t), torch.zeros_like(t)
        for m in range(1, len(a) + 1):
            cm, sm = torch.cos(m * t), torch.sin(m * t)
            r = r + float(a[m - 1]) * cm + float(b[m - 1]) * sm
            dr = dr + m * (-float(a[m - 1]) * sm + float(b[m - 1]) * cm)
            ddr = ddr - m * m * (float(a[m - 1]) * cm + float(b[m - 1]) * sm)
        return (r * c, r * s), (dr * c - r * s, dr * s + r * c), (ddr * c - 2 * dr * s - r * c, ddr * s + 2 * dr * c - r * s)
    if case["curve"] == "circle":
        return (c, s), (-s, c), (-c, -s)
    c2, s2 = torch.cos(2 * t), torch.sin(2 * t)
    return (c + 0.65 * c2 - 0.65, 1.5 * s), (-s - 1.3 * s2, 1.5 * c), (-c - 2.6 * c2, -1.5 * s)


def _bessel(z):
    return torch.special.bessel_j0(z), torch.special.bessel_y0(z), torch.special.bessel_j1(z), torch.special.bessel_y1(z)


class _Nystrom:
    """The operator on the uniform grid of nq points, at targets t = 2 pi p / groups + delta_q
    (groups divides nq)."""

    def __init__(self, case, k, form, nq, star=None):
        self.case, self.k, self.form, self.nq, self.star = case, k, form, nq, star
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.t = torch.arange(nq, dtype=torch.float64, device=self.dev) * (2 * math.pi / nq)
        (self.x, self.y), (self.xp, self.yp), (self.xpp, self.ypp) = _curve(case, self.t, star)
        self.sp = torch.sqrt(self.xp ** 2 + self.yp ** 2)

    def _log_weights(self, delta):
        """R(delta - 2 pi j / nq): Kress's weights of ln(4 sin^2(./2)), from one FFT"""
        n = self.nq // 2
        c = torch.zeros(self.nq, dtype=torch.complex128, device=self.dev)
        m = torch.arange(1, n, dtype=torch.float64, device=self.dev)
        c[1:n] = torch.polar(-(2 * math.pi / n) / m, m * delta)
        c[n] = -(math.pi / n ** 2) * complex(math.cos(n * delta), math.sin(n * delta))
        return torch.fft.fft(c).real

    def rows(self, groups, p0, p1, delta):
        """matrix rows of the targets p0 <= p < p1 at offset delta (without the jump term)"""
        nq, k, dev = self.nq, self.k, self.dev
        step = nq // groups
        p = torch.arange(p0, p1, device=dev)
        j = (torch.arange(nq, device=dev)[None, :] - step * p[:, None]) % nq
        R = self._log_weights(delta)[j]
        half = torch.sin(0.5 * (delta - torch.arange(nq, dtype=torch.float64, device=dev) * (2 * math.pi / nq)))
        hit = (half.abs() < 1e-9)[j]
        lg = torch.log(4 * half.square().clamp_min(1e-300))[j]
        del j
        (tx, ty), _, _ = _curve(self.case, 2 * math.pi / groups * p.double() + delta, self.star)
        dx, dy = tx[:, None] - self.x[None, :], ty[:, None] - self.y[None, :]
        r = torch.sqrt(dx * dx + dy * dy)
        r[hit] = 1.0
        j0, y0, j1, y1 = _bessel(k * r)
        sp = self.sp[None, :]
        m1 = -j0 * sp / (4 * math.pi)
        m2r = -0.25 * y0 * sp - m1 * lg                      # (i/4) H0 |x'| = (-Y0 + i J0) |x'| / 4
        m2i = 0.25 * j0 * sp
        euler = 0.57721566490153286
        d = (-euler / (2 * math.pi) - torch.log(0.5 * k * self.sp) / (2 * math.pi)) * self.sp
        m2r = torch.where(hit, d[None, :].expand_as(m2r), m2r)
        m2i = torch.where(hit, (0.25 * sp).expand_as(m2i), m2i)
        m1 = torch.where(hit, (-sp / (4 * math.pi)).expand_as(m1), m1)
        w = math.pi * 2 / nq
        S = torch.complex(R * m1 + w * m2r, w * m2i)
        if self.form != "combined":
            return S
        q = (dx * self.yp[None, :] - dy * self.xp[None, :]) / r
        l1 = -(k / (4 * math.pi)) * j1 * q
        l2r = -0.25 * k * y1 * q - l1 * lg                   # (i k / 4) H1 q = (-Y1 + i J1) k q / 4
        l2i = 0.25 * k * j1 * q
        d = (self.xpp * self.yp - self.ypp * self.xp) / (4 * math.pi * self.sp ** 2)
        l2r = torch.where(hit, d[None, :].expand_as(l2r), l2r)
        l2i = torch.where(hit, torch.zeros_like(l2i), l2i)
        l1 = torch.where(hit, torch.zeros_like(l1), l1)
        K = torch.complex(R * l1 + w * l2r, w * l2i)
        return K - 1j * k * S                                # eta = k

    def apply(self, phi, groups, deltas):
        """[nrhs][groups * len(deltas)]: the integral at every target, deltas fastest"""
        out = torch.empty(phi.shape[0], groups, len(deltas), dtype=torch.complex128, device=self.dev)
        n = max(1, (1 << 24) // self.nq)
        for q, delta in enumerate(deltas):
            for p0 in range(0, groups, n):
                p1 = min(groups, p0 + n)
                out[:, p0:p1, q] = (self.rows(groups, p0, p1, delta) @ phi.T).T
        return out.reshape(phi.shape[0], -1)

    def solve(self, rhs):
        """the density on the grid: (1/2 I + K - i eta S) phi = rhs"""
        A = torch.empty(self.nq, self.nq, dtype=torch.complex128, device=self.dev)
        n = max(1, (1 << 24) // self.nq)
        for p0 in range(0, self.nq, n):
            A[p0:p0 + n] = self.rows(self.nq, p0, min(self.nq, p0 + n), 0.0)
        A.diagonal().add_(0.5)
        return torch.linalg.solve(A, rhs)

    def resample(self, phi, groups, deltas):
        """the trigonometric interpolant of phi at the targets, deltas fastest"""
        c = torch.fft.fft(phi)
        m = torch.fft.fftfreq(self.nq, 1.0 / self.nq, dtype=torch.float64, device=self.dev)
        out = torch.empty(groups, len(deltas), dtype=torch.complex128, device=self.dev)
        for q, delta in enumerate(deltas):
            out[:, q] = torch.fft.ifft(c * torch.polar(torch.ones_like(m), m * delta))[:: self.nq // groups]
        return out.reshape(-1)


def _offsets(patches, Np):
    """parameter offsets of a patch's Fejer nodes from its start, in the package's point order"""
    z = np.cos(np.pi * (2 * np.arange(Np) + 1) / (2 * Np))
    return [float(v) for v in (math.pi / patches) * (1.0 + z)]


def _grid(patches, k):
    """points of the uniform grid: a multiple of the patches, above twice the bandwidth of kernel times density"""
    m = max(2, int(math.ceil(max(9.6 * k, 400.0) / patches)))
    return patches * (m + m % 2)


def exact(case, seed):
    op = case["op"]
    if op == "group":
        out = []
        for a, b, k, patches, ang in _stars(case, seed):
            nq = _grid(patches, k)
            N = _Nystrom(case, k, "combined", nq, star=(a, b))
            ph = k * (math.cos(ang) * N.x + math.sin(ang) * N.y)
            phi = N.solve(-torch.complex(torch.cos(ph), torch.sin(ph)))
            out.append(N.resample(phi, patches, _offsets(patches, case["Np"])))
        return torch.cat(out).cpu().numpy()
    k, patches = case["k"], case["patches"]
    if k > 2500.0:
        return None                  # the dense operator takes longer than its use is worth
    nq, deltas = _grid(patches, k), _offsets(patches, case["Np"])
    N = _Nystrom(case, k, case["form"], nq)
    if op in ("solve", "solve_spectral"):
        if nq > 13000:
            return None
        a = _angle(seed)
        ph = k * (math.cos(a) * N.x + math.sin(a) * N.y)
        phi = N.solve(-torch.complex(torch.cos(ph), torch.sin(ph)))
        return N.resample(phi, patches, deltas).cpu().numpy()
    nrhs = case.get("nrhs", 1)
    phi = _density(case, seed, N.x, N.y, nrhs)
    if op == "field":
        tx, ty = (torch.from_numpy(v).to(N.dev) for v in _targets(case, seed))
        out = []
        for i in range(0, tx.numel(), max(1, (1 << 24) // nq)):
            dx = tx[i:i + max(1, (1 << 24) // nq), None] - N.x[None, :]
            dy = ty[i:i + max(1, (1 << 24) // nq), None] - N.y[None, :]
            r = torch.sqrt(dx * dx + dy * dy)
            j0, y0, j1, y1 = _bessel(k * r)
            ker = torch.complex(-0.25 * y0, 0.25 * j0) * N.sp
            if case["form"] == "combined":
                q = (dx * N.yp - dy * N.xp) / r
                ker = torch.complex(-0.25 * k * y1 * q, 0.25 * k * j1 * q) - 1j * k * ker
            out.append((2 * math.pi / nq) * (ker @ phi[0]))
        return torch.cat(out).cpu().numpy()
    y = N.apply(phi, patches, deltas)
    if case["form"] == "combined":
        t = (2 * math.pi / patches) * torch.arange(patches, dtype=torch.float64, device=N.dev)[:, None] + \
            torch.tensor(deltas, dtype=torch.float64, device=N.dev)[None, :]
        (x1, x2), _, _ = _curve(case, t.reshape(-1))
        y = y + 0.5 * _density(case, seed, x1, x2, nrhs)
    if op == "host":
        return y[0].cpu().numpy()
    return y if op in ("batch", "batch_mixed") else y[0]
