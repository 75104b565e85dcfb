"""The work that users of this framework have it do, as cases that can be measured.

A pipe is a spectral velocity state (NR radial points, NT theta slots, NZ axial modes).
Four kinds of call:

  step       device-resident states are handed over, advanced a number of time steps and
             read back, as a program does that couples the stepper with other device code
             (edge tracking, Newton-Krylov solvers, data collection);
  host       the same with the states of the whole ensemble in pinned host memory, one call
             per time step (nsp_step_host);
  sample     the diagnostics of every member between two stretches of steps: friction,
             divergence, mean profiles, cross sections;
  nonlinear  the nonlinear term of one explicit field.

States are Hagen-Poiseuille flow plus a seeded divergence-free perturbation whose spectrum
decays towards the cut-off.
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "nspipe-gpu_gb300"))

PI2 = 6.283185307179586
D_IM, TOL, MAXIT, QDES = 0.51, 5e-8, 10, 0.5
# The uneven batch: three resolutions, each with a range of Reynolds numbers.
UNEVEN = ((16, 48, 32, 65, 2000.0, 2400.0), (8, 64, 48, 129, 2400.0, 3000.0), (4, 96, 96, 193, 3000.0, 4000.0))


def _case(name, kind, precision, members, NR, NT, NZ, Re=2000.0, Re1=0.0, dt=0.01, LZ=2 * PI2, amp=1e-3, steps=1,
          uneven=False):
    return {"name": name, "kind": kind, "precision": precision, "members": members, "NR": NR, "NT": NT, "NZ": NZ,
            "Re": Re, "Re1": Re1 or Re, "dt": dt, "LZ": LZ, "amp": amp, "steps": steps, "uneven": uneven}


def listed():
    return [
        # one small transitional pipe, one step at a time: latency and launches count
        _case("one_mixed", "step", "mixed", 1, 48, 32, 65),
        # the same in the plain form, the drop-in replacement of the reference
        _case("one_fp64", "step", "fp64", 1, 48, 32, 65),
        # the batched ensemble that the headline is quoted on
        _case("ensemble_mixed", "step", "mixed", 64, 48, 32, 65, steps=8),
        # an ensemble in the plain form
        _case("ensemble_fp64", "step", "fp64", 16, 48, 32, 65, steps=2),
        # pipes of three resolutions and 28 Reynolds numbers stepped together
        _case("uneven_mixed", "step", "mixed", 28, 48, 32, 65, dt=0.006, amp=5e-3, steps=2, uneven=True),
        # one turbulent pipe at full resolution
        _case("turbulent_mixed", "step", "mixed", 1, 96, 128, 257, Re=5300.0, dt=0.002, amp=8e-3, steps=3),
        # the reference's default set-up, plain form
        _case("default_fp64", "step", "fp64", 1, 48, 64, 257, Re=1850.0, LZ=100.0, steps=1),
        # a few pipes of an odd radial size and of transform lengths that are no powers of two
        _case("ragged_mixed", "step", "mixed", 7, 61, 36, 55, Re=2300.0, Re1=2600.0, dt=0.008, amp=5e-3, steps=3),
        # the ensemble with its states in host memory at every step
        _case("host_mixed", "host", "mixed", 64, 48, 32, 65),
        # diagnostics of the ensemble, taken every few dozen steps
        _case("sample_ensemble", "sample", "mixed", 64, 48, 32, 65),
        # the nonlinear term as an operator of a user's own solver
        _case("nonlinear_fp64", "nonlinear", "fp64", 1, 64, 48, 129, Re=2700.0, amp=0.02),
    ]


def draw(rng):
    kind, precision = rng.choice([("step", "mixed"), ("step", "mixed"), ("step", "mixed"), ("step", "fp64"),
                                  ("step", "fp64"), ("host", "mixed"), ("sample", "mixed"), ("nonlinear", "fp64")])
    NR = int(round(math.exp(rng.uniform(math.log(24), math.log(97)))))
    NT = rng.choice([16, 24, 32, 32, 36, 48, 64, 96])
    NZ = rng.choice([17, 25, 33, 49, 55, 65, 97, 129, 193])
    S = NR * NT * NZ
    cap = {"step": 6.0e6 if precision == "mixed" else 1.2e6, "host": 6.0e6, "sample": 6.0e6, "nonlinear": 1.2e6}[kind]
    while S > cap:
        NZ = rng.choice([17, 25, 33, 49, 55])
        NT = min(NT, 48)
        S = NR * NT * NZ
    most = max(1, min(64, int(cap / S)))
    members = 1 if kind == "nonlinear" else int(round(math.exp(rng.uniform(0.0, math.log(most)))))
    Re = float(rng.randint(1800, 3600))
    c = _case("", kind, precision, members, NR, NT, NZ, Re=Re, Re1=Re + rng.choice([0, 0, 25 * members]),
              dt=round(0.16 / max(NT, 16) + rng.uniform(-1e-4, 1e-4), 6), LZ=rng.choice([1, 2, 4]) * PI2,
              amp=round(math.exp(rng.uniform(math.log(1e-3), math.log(4e-3))), 5),
              steps=rng.randint(1, 4) if kind == "step" else 1)
    del c["name"]
    return c


def _groups(case):
    """[(NR, NT, NZ, [Re of each member])] in member order."""
    if case["uneven"]:
        rows = UNEVEN
    else:
        rows = ((case["members"], case["NR"], case["NT"], case["NZ"], case["Re"], case["Re1"]),)
    return [(nr, nt, nz, [a + (b - a) * k / max(n - 1, 1) for k in range(n)]) for n, nr, nt, nz, a, b in rows]


def _grid(NR):
    """The wall-clustered radial grid."""
    n_p = NR + int(math.sqrt(float(NR)))
    i = np.arange(n_p - NR, n_p)
    r = 0.5 * (1.0 + np.cos(0.5 * PI2 * ((n_p - i - 1) / float(n_p))))
    for _ in range(10):
        dr = 1.5 * r[0] - 0.5 * r[1]
        r = r * (1.0 + dr) - dr
    return r


def _fields(case, seed, dev):
    """Per group a complex128 tensor (members, 3, NR, NT, NZ): u_r, u_theta, u_z.

    The curls of psi e_z and chi e_theta, psi = a (1-r^2)^2 r^|m|, chi = b (1-r^2)^2 r^(|m|+1), plus the base
    flow 1 - r^2; the largest coefficient of the perturbation is amp times 1 to 1.6 from member to member."""
    gen = torch.Generator().manual_seed(seed)
    out = []
    for NR, NT, NZ, res in _groups(case):
        M = len(res)
        r = torch.from_numpy(_grid(NR)).to(dev).view(NR, 1, 1)
        m = torch.tensor([t if t < NT // 2 else t - NT for t in range(NT)], dtype=torch.float64)
        k = torch.arange(NZ, dtype=torch.float64)
        decay = torch.exp(-m.abs().view(NT, 1) / max(1.0, NT / 16.0) - k.view(1, NZ) / max(1.0, NZ / 16.0))
        decay[NT // 2] = 0.0
        decay[:, NZ - 1] = 0.0
        ab = torch.randn((2, M, NT, NZ, 2), generator=gen, dtype=torch.float64)
        ab = torch.view_as_complex(ab) * decay
        for t in range(1, NT // 2):  # the k_z = 0 plane of a real field
            ab[:, :, NT - t, 0] = ab[:, :, t, 0].conj()
        ab[:, :, 0, 0] = 0.0
        a, b = (x.to(dev).view(M, 1, NT, NZ) for x in ab)
        n, mm = m.abs().to(dev).view(1, NT, 1), m.to(dev).view(1, NT, 1)
        kz = (k.to(dev) * (PI2 / case["LZ"])).view(1, 1, NZ)
        one = 1.0 - r * r
        rn1 = torch.where(n > 0, r ** (n - 1.0).clamp(min=0.0), torch.zeros_like(r * n))
        u = torch.empty((M, 3, NR, NT, NZ), dtype=torch.complex128, device=dev)
        u[:, 0] = 1j * mm * a * (one ** 2 * rn1) - 1j * kz * b * (one ** 2 * r ** (n + 1.0))
        u[:, 1] = -a * (n * rn1 * one ** 2 - 4.0 * r ** (n + 1.0) * one)
        u[:, 2] = b * ((n + 2.0) * r ** n * one ** 2 - 4.0 * r ** (n + 2.0) * one)
        size = torch.tensor([case["amp"] * (1.0 + 0.6 * j / M) for j in range(M)], device=dev, dtype=torch.float64)
        u *= (size / u.abs().reshape(M, -1).amax(1)).view(M, 1, 1, 1, 1)
        u[:, 2, :, 0, 0] += one.view(1, NR)
        out.append(u)
    return out


def prepare(case, seed):
    import nspipe_gb300 as nsp
    dev = torch.device("cuda", 0)
    prm = [nsp.make_params(nr, nt, nz, re, case["dt"], case["LZ"], d_im=D_IM, maxit=MAXIT, tol=TOL, Qdes=QDES)
           for nr, nt, nz, res in _groups(case) for re in res]
    st = nsp.Stepper(prm, precision=nsp.NSP_MIXED if case["precision"] == "mixed" else nsp.NSP_FP64, device=0)
    u = _fields(case, seed, dev)
    s = {"case": case, "stepper": st}
    if case["kind"] == "host":
        flat = torch.cat([x.reshape(-1) for x in u])
        s["in"] = torch.empty(flat.shape, dtype=flat.dtype, pin_memory=True).copy_(flat).numpy()
        s["out"] = torch.empty(flat.shape, dtype=flat.dtype, pin_memory=True).numpy()
        s["out"][:] = 0
        return s
    s["u"] = u
    s["out"] = [torch.zeros_like(x) for x in u]
    torch.cuda.synchronize()
    if case["kind"] == "sample":
        _hand_over(s)
    return s


def _hand_over(s):
    m = 0
    for g in s["u"]:
        for x in g:
            s["stepper"].set_state_device(m, x[0], x[1], x[2])
            m += 1


def run(s):
    st, case = s["stepper"], s["case"]
    if case["kind"] == "host":
        out, iters = st.step_host(case["steps"], s["in"], s["out"])
        return {"u": out, "iterations": iters}
    if case["kind"] == "nonlinear":
        st.nonlinear(0, list(s["u"][0][0]), list(s["out"][0][0]))
        return s["out"]
    if case["kind"] == "sample":
        d = st.diag_all()
        mean = st.mean_profile_all()
        q, w = st.cross_sections_all()
        return {"diag": np.array([[x.u_centre, x.u_tau, x.flux, x.re_tau, x.div_max, x.div_wall] for x in d]),
                "mean": np.concatenate(mean), "q": np.concatenate(q), "u": np.concatenate(w)}
    _hand_over(s)
    iters = st.step(case["steps"])
    m = 0
    for g in s["out"]:
        for x in g:
            st.get_state_device(m, x[0], x[1], x[2])
            m += 1
    return {"u": s["out"], "iterations": iters}


def work(case):
    """States in and out once per step (once per call for operators and diagnostics), and the operations of the
    transforms, products, stencils and banded solves of one predictor and one corrector pass per step."""
    nbytes = flops = 0.0
    for NR, NT, NZ, res in _groups(case):
        M, S, NTP, NZR = len(res), NR * NT * NZ, 3 * NT // 2, 3 * (NZ - 1)
        inverse = 9 * NR * NZ * 5 * NTP * math.log2(NTP) + 12 * NR * NTP * 2.5 * NZR * math.log2(NZR)
        forward = 3 * NR * NZ * 5 * NTP * math.log2(NTP) + 3 * NR * NTP * 2.5 * NZR * math.log2(NZR)
        nl = inverse + forward + 22.0 * NR * NTP * NZR + 3 * 28.0 * S
        if case["kind"] in ("step", "host"):
            nbytes += case["steps"] * M * 96.0 * S
            flops += case["steps"] * M * 2 * (nl + 250.0 * S)
        elif case["kind"] == "nonlinear":
            nbytes += 96.0 * S
            flops += nl
        else:
            nbytes += M * (48.0 * S + 8.0 * (NR + 2 * NZR + 6))
            flops += M * (3 * NR * NT * 5 * NZR * math.log2(NZR) + 40.0 * S)
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------- the same in 64 bits, plainly

def _weights(z, x, m):
    """Finite-difference weights of the derivatives 0..m at z on the points x (Fornberg, SIAM Review 40, 1998)."""
    n = len(x)
    c = np.zeros((m + 1, n))
    c[0, 0], c1, c4 = 1.0, 1.0, x[0] - z
    for i in range(1, n):
        top, c2, c5, c4 = min(i, m), 1.0, c4, x[i] - z
        for j in range(i):
            c3 = x[i] - x[j]
            c2 *= c3
            if j == i - 1:
                for k in range(top, 0, -1):
                    c[k, i] = c1 * (k * c[k - 1, i - 1] - c5 * c[k, i - 1]) / c2
                c[0, i] = -c1 * c5 * c[0, i - 1] / c2
            for k in range(top, 0, -1):
                c[k, j] = (c4 * c[k, j] - k * c[k - 1, j]) / c3
            c[0, j] = c4 * c[0, j] / c3
        c1 = c2
    return c


class _Pipe:
    """The discrete operators of one resolution: 7-point radial differences with even / odd folding at the axis."""

    def __init__(self, NR, NT, NZ, res, case, dev):
        self.NR, self.NT, self.NZ, self.NTP, self.NZR, self.dev = NR, NT, NZ, 3 * NT // 2, 3 * (NZ - 1), dev
        r = _grid(NR)
        ext = np.concatenate([-r[2::-1], r])
        D, D2, rdr = np.zeros((2, NR, NR)), np.zeros((2, NR, NR)), np.zeros(NR)
        for i in range(NR):
            cols = np.arange(i, min(i + 6, NR + 2) + 1)
            w = _weights(ext[i + 3], ext[cols], len(cols) - 1)
            at = np.where(cols < 3, 2 - cols, cols - 3)  # a point left of the axis stands for its mirror image
            for sign in (0, 1):
                f = np.where((cols < 3) & (sign == 1), -1.0, 1.0)
                np.add.at(D[sign, i], at, f * w[1])
                np.add.at(D2[sign, i], at, f * w[2])
            up, dn = (r[i + 1] if i < NR - 1 else r[i]) - r[i], (r[i - 1] if i else 0.0) - r[i]
            for k in range(len(cols)):  # the Taylor expansion at r_i over its two neighbours' interval
                np.add.at(rdr, at, (up ** (k + 1) - dn ** (k + 1)) / math.factorial(k + 1) * r[i] * w[k])
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
        self.D, self.r, self.rdr = t(D), t(r), t(rdr)
        self.axis = t(_weights(0.0, r[:4], 0)[0])
        self.ri = (1.0 / self.r).view(NR, 1, 1)
        m = torch.tensor([k if k < NT // 2 else k - NT for k in range(NT)], device=dev)
        self.odd = m % 2 != 0
        self.kt = m.double().view(1, NT, 1)
        self.kz = (torch.arange(NZ, device=dev, dtype=torch.float64) * (PI2 / case["LZ"])).view(1, 1, NZ)
        self.re = torch.tensor(res, device=dev, dtype=torch.float64).view(-1, 1, 1, 1)
        self.dt = case["dt"]
        L = D2 + D / r.reshape(1, NR, 1)
        L[:, -1] = 0.0  # the wall row of the Laplacian is the wall value itself
        L[:, -1, -1] = 1.0
        self.L = t(L)

    def table(self, T, u, flag):
        """T[parity] applied along r; flag 1: u_r, u_theta; 0: u_z, p."""
        out = torch.empty_like(u)
        for par in (0, 1):
            at = self.odd if par else ~self.odd
            x = u[..., at, :]
            out[..., at, :] = torch.einsum("ij,...jtl->...itl", T[abs(par - flag)].to(u.dtype), x)
        return out

    def nonlinear(self, u):
        """-(u.grad)u on the 3/2-dealiased grid, and the wall-shear forcing of the mean axial mode."""
        NT, NTP, NZ, NZR = self.NT, self.NTP, self.NZ, self.NZR

        def phys(x):
            full = x.new_zeros(x.shape[:-2] + (NTP, NZR // 2 + 1))
            full[..., : NT // 2, :NZ] = x[..., : NT // 2, :]
            full[..., NTP - NT // 2:, :NZ] = x[..., NT // 2:, :]
            return torch.fft.irfft(torch.fft.ifft(full, dim=-2, norm="forward"), n=NZR, dim=-1, norm="forward")

        p = [phys(u[:, c]) for c in range(3)]
        n = [0.0, 0.0, 0.0]
        for c in range(3):
            n[c] = -(p[0] * phys(self.table(self.D, u[:, c], 1 if c < 2 else 0))
                     + p[1] * phys(1j * self.kt * self.ri * u[:, c]) + p[2] * phys(1j * self.kz * u[:, c]))
        n[0] = n[0] + p[1] * p[1] * self.ri
        n[1] = n[1] - p[0] * p[1] * self.ri
        out = torch.zeros_like(u)
        for c in range(3):
            h = torch.fft.fft(torch.fft.rfft(n[c], dim=-1), dim=-2) / (NTP * NZR)
            out[:, c, :, : NT // 2, : NZ - 1] = h[..., : NT // 2, : NZ - 1]
            out[:, c, :, NT // 2 + 1:, : NZ - 1] = h[..., NTP - NT // 2 + 1:, : NZ - 1]
        wall = (self.D[0, -1] * u[:, 2, :, 0, 0].real).sum(-1)
        out[:, 2, :, 0, 0] -= (2.0 / self.re.view(-1) * wall).view(-1, 1)
        return out

    def factor(self, rows):
        """LU factors, in place, of a banded matrix rows[NR][7] of tensors (no pivoting)."""
        for i in range(self.NR):
            for d in (3, 2, 1):
                if i - d >= 0:
                    f = rows[i][3 - d] / rows[i - d][3]
                    rows[i][3 - d] = f
                    for t in range(1, 4):
                        if i - d + t < self.NR:
                            rows[i][3 - d + t] = rows[i][3 - d + t] - f * rows[i - d][3 + t]
        return rows

    def solve(self, rows, b):
        x = list(b.unbind(1))
        for i in range(self.NR):
            for d in range(1, min(3, i) + 1):
                x[i] = x[i] - rows[i][3 - d] * x[i - d]
        for i in reversed(range(self.NR)):
            for d in range(1, min(3, self.NR - 1 - i) + 1):
                x[i] = x[i] - rows[i][3 + d] * x[i + d]
            x[i] = x[i] / rows[i][3]
        return torch.stack(x, 1)

    def operators(self):
        NR, NT, NZ = self.NR, self.NT, self.NZ
        r2 = (self.r ** -2).view(NR, 1, 1)
        base = -self.kz ** 2 - self.kt ** 2 * r2
        self.diag = [base - r2 - 2.0 * self.kt * r2, base - r2 + 2.0 * self.kt * r2, base]
        odd = self.odd.view(1, NT, 1)
        zero = torch.zeros((1, NT, NZ), device=self.dev, dtype=torch.float64)
        c = (D_IM / self.re).view(-1, 1, 1)

        def banded(T, flag, diag, wall, helmholtz):
            rows = []
            for i in range(NR):
                row = []
                for e in range(7):
                    j = i + e - 3
                    v = zero
                    if 0 <= j < NR:
                        v = torch.where(odd, T[abs(1 - flag), i, j], T[abs(0 - flag), i, j]) + zero
                        if i == NR - 1:
                            v = wall(j) + zero
                        else:
                            v = v + diag[i] if e == 3 else v
                            v = (1.0 / self.dt if e == 3 else 0.0) - c * v if helmholtz else v
                    row.append(v)
                rows.append(row)
            return self.factor(rows)

        eye = lambda j: 1.0 if j == NR - 1 else 0.0  # noqa: E731
        mean = torch.zeros((1, NT, NZ), device=self.dev, dtype=torch.bool)
        mean[0, 0, 0] = True
        slope = lambda j: torch.where(mean, torch.tensor(eye(j), device=self.dev, dtype=torch.float64),  # noqa: E731
                                      torch.where(odd, self.D[1, -1, j], self.D[0, -1, j]))
        self.H = [banded(self.L, 1, self.diag[0], eye, True), banded(self.L, 1, self.diag[1], eye, True),
                  banded(self.L, 0, self.diag[2], eye, True)]
        self.P = banded(self.L, 0, self.diag[2], slope, False)
        # a unit of wall divergence, made of wall values of u+, u-, u_z and of a pressure with p_wall = -1
        unit = torch.zeros((self.re.numel(), NR, NT, NZ), device=self.dev, dtype=torch.complex128)
        unit[:, -1] = 1.0
        h = [self.solve(self.H[k], unit) for k in range(3)]
        g = self.grad(self.solve(self.P, -unit))
        g = [g[0] + 1j * g[1], g[0] - 1j * g[1], g[2]]
        v = [g[k] - g[k][:, -1:] * h[k] for k in range(3)]
        s = self.wall_div(v)
        s[:, 0, 0] = 1.0
        v = torch.stack([x / s.unsqueeze(1) for x in v], 1)
        v[..., 0, 0] = 0.0
        self.V = v
        one = torch.ones((self.re.numel(), NR, NT, NZ), device=self.dev, dtype=torch.complex128)
        one[:, -1] = 0.0
        self.uc = self.solve(self.H[2], one)[..., 0, 0].real
        self.Qc = (self.uc * self.rdr).sum(-1, keepdim=True)

    def grad(self, p):
        return [self.table(self.D, p, 0), 1j * self.kt * self.ri * p, 1j * self.kz * p]

    def div(self, u):
        return self.table(self.D, u[0], 1) + (u[0] + 1j * self.kt * u[1]) * self.ri + 1j * self.kz * u[2]

    def wall_div(self, v):
        """d_r u_r + u_r + i k_theta u_theta + i k_z u_z at the wall, of (u+, u-, u_z)."""
        return self.div([0.5 * (v[0] + v[1]), -0.5j * (v[0] - v[1]), v[2]])[:, -1]

    def explicit(self, u):
        c = (1.0 - D_IM) / self.re
        pm = [u[:, 0] + 1j * u[:, 1], u[:, 0] - 1j * u[:, 1], u[:, 2]]
        e = [x / self.dt + c * (self.table(self.L, x, 1 if k < 2 else 0) + self.diag[k] * x) for k, x in enumerate(pm)]
        return torch.stack([0.5 * (e[0] + e[1]), -0.5j * (e[0] - e[1]), e[2]], 1)

    def advance(self, rhs):
        d = self.div([rhs[:, 0], rhs[:, 1], rhs[:, 2]])
        d[:, -1] = 0.0
        g = self.grad(self.solve(self.P, d))
        f = [rhs[:, k] - g[k] for k in range(3)]
        v = [f[0] + 1j * f[1], f[0] - 1j * f[1], f[2]]
        for k in range(3):
            v[k][:, -1] = 0.0
            v[k] = self.solve(self.H[k], v[k])
        s = self.wall_div(v).unsqueeze(1)
        v = [v[k] - s * self.V[:, k] for k in range(3)]
        u = torch.stack([0.5 * (v[0] + v[1]), -0.5j * (v[0] - v[1]), v[2]], 1)
        u[:, 0, :, 0, 0] = 0.0
        u[:, 1:, :, 0, 0] = u[:, 1:, :, 0, 0].real.to(u.dtype)
        q = (u[:, 2, :, 0, 0].real * self.rdr).sum(-1, keepdim=True)
        u[:, 2, :, 0, 0] += (QDES - q) / self.Qc * self.uc
        return u

    def steps(self, u, n):
        self.operators()
        sq = lambda x: (x.real ** 2 + x.imag ** 2).reshape(x.shape[0], -1).amax(1)  # noqa: E731
        for _ in range(n):
            old = self.nonlinear(u)
            e = self.explicit(u)
            it = self.advance(old + e)
            going = torch.ones(u.shape[0], dtype=torch.bool, device=self.dev)
            for _k in range(MAXIT):
                new = self.advance(D_IM * self.nonlinear(it) + (1.0 - D_IM) * old + e)
                err = sq(it - new) / sq(it)
                it = torch.where(going.view(-1, 1, 1, 1, 1), new, it)
                going = going & (err > TOL)
                if not bool(going.any()):
                    break
            u = it
        return u

    def diagnostics(self, u):
        m = u[:, 2, :, 0, 0].real
        tau = torch.sqrt((m * self.D[0, -1]).sum(-1).abs() / self.re.view(-1))
        d = self.div([u[:, 0], u[:, 1], u[:, 2]]).abs()
        diag = torch.stack([(m[:, :4] * self.axis).sum(-1), tau, (m * self.rdr).sum(-1), tau * self.re.view(-1),
                            d[:, :-1].reshape(len(u), -1).amax(1), d[:, -1].reshape(len(u), -1).amax(1)], 1)
        full = u.new_zeros(u.shape[:-2] + (self.NTP, self.NZR // 2 + 1))
        full[..., : self.NT // 2, : self.NZ] = u[..., : self.NT // 2, :]
        full[..., self.NTP - self.NT // 2:, : self.NZ] = u[..., self.NT // 2:, :]
        p = torch.fft.irfft(torch.fft.ifft(full, dim=-2, norm="forward"), n=self.NZR, dim=-1, norm="forward")
        sq = (p * p).mean(-2)  # (members, 3, NR, NZR)
        w = self.rdr.view(1, -1, 1)
        return diag, m, ((sq[:, 0] + sq[:, 1]) * w).sum(1), (sq[:, 2] * w).sum(1)


def exact(case, seed):
    dev = torch.device("cuda", 0) if torch.cuda.is_available() else torch.device("cpu")
    u = _fields(case, seed, dev)
    pipes = [_Pipe(nr, nt, nz, res, case, dev) for nr, nt, nz, res in _groups(case)]
    if case["kind"] == "nonlinear":
        return [pipes[0].nonlinear(u[0])]
    if case["kind"] == "sample":
        part = [[], [], [], []]
        for p, x in zip(pipes, u):
            for k in range(0, len(x), 8):  # a few members at a time
                p.re = torch.tensor(_groups(case)[0][3][k: k + 8], device=dev, dtype=torch.float64).view(-1, 1, 1, 1)
                for at, v in zip(part, p.diagnostics(x[k: k + 8])):
                    at.append(v.cpu())
        diag, mean, q, w = (torch.cat(v).numpy() for v in part)
        return {"diag": diag, "mean": mean.reshape(-1), "q": q.reshape(-1), "u": w.reshape(-1)}
    out = []
    for (nr, nt, nz, res), x in zip(_groups(case), u):
        done = []
        for k in range(0, len(x), 8):
            done.append(_Pipe(nr, nt, nz, res[k: k + 8], case, dev).steps(x[k: k + 8], case["steps"]))
        out.append(torch.cat(done))
    if case["kind"] == "host":
        return {"u": torch.cat([x.reshape(-1) for x in out]).cpu().numpy(), "iterations": None}
    return {"u": out, "iterations": None}
