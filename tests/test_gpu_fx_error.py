"""The FP64 form's transforms against extended precision: the nonlinear term of one level within
5e-16 of its norm.

With u_r = 0 the term needs no radial derivative, so the levels are apart and one of them is
evaluated in long double (64 bits of mantissa or more) by sums over the modes:
    N_r = u_t u_t / r,  N_t = -(u_t d_t u_t / r + u_z d_z u_t),  N_z = -(u_t d_t u_z / r + u_z d_z u_z)
(d_t, d_z: derivatives along the two periodic directions; the mean axial mode, which carries the
wall forcing, is left out).

Tolerance: the fixed-point transforms leave 2^-55 of a line's norm or less, one after the other along
the two directions and back; what is computed in FP64 around them -- the factors i m, i k_z and 1/r,
the values in and out of the three stages, the products and sums -- is about ten roundings of some
6e-17 each.  In quadrature 2.2e-16; 5e-16 is twice that (eight bits lost in a scale or a product
would be 1e-14)."""
import numpy as np
import pytest

from conftest import PI2
from test_gpu_fx_transforms import LZ, Re, nonlinear, rough_field
from test_gpu_parity import nsp  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu

NR, LEVEL = 9, 5
L = np.longdouble


def roots(n):
    """exp(2 pi i e / n), e < n, to long double's rounding: angles reduced to an eighth of a turn."""
    pi = L("3.14159265358979323846264338327950288")
    e = np.arange(n)
    q, rest = 4 * e // n, 4 * e % n  # quarter turn and angle within it, (pi/2) rest / n
    near = 2 * rest <= n
    x = pi * L(0.5) * np.where(near, rest, n - rest).astype(L) / L(n)
    c, s = np.where(near, np.cos(x), np.sin(x)), np.where(near, np.sin(x), np.cos(x))
    re = np.choose(q, [c, -s, -c, s])
    im = np.choose(q, [s, c, -s, -c])
    return re, im


def matmul(a, b):
    """(re, im) pairs."""
    return a[0] @ b[0] - a[1] @ b[1], a[0] @ b[1] + a[1] @ b[0]


def reference(u, r, NT, NZ):
    """(N_r, N_t, N_z) of one level as complex long double parts; u: u_t, u_z of that level."""
    NTP, NZR = 3 * NT // 2, 3 * (NZ - 1)
    m = np.array([t if t < NT // 2 else t - NT for t in range(NT)])
    l = np.arange(NZ)
    wt, wz = roots(NTP), roots(NZR)
    at, az = np.outer(np.arange(NTP), m) % NTP, np.outer(l, np.arange(NZR)) % NZR
    T, Z = (wt[0][at], wt[1][at]), (wz[0][az], wz[1][az])
    kz = l.astype(L) * (L(PI2) / L(LZ))

    def phys(re, im):
        g = matmul(T, (re, im))
        two = np.where(l == 0, L(1), L(2))
        return (two * g[0]) @ Z[0] - (two * g[1]) @ Z[1]

    f = []
    for a in u:
        re, im = a.real.astype(L), a.imag.astype(L)
        mm = m.astype(L).reshape(-1, 1)
        f.append((phys(re, im), phys(-mm * im, mm * re) / r, phys(-kz * im, kz * re)))
    (t, tt, tz), (z, zt, zz) = f
    out = []
    for n in (t * t / r, -(t * tt + z * tz), -(t * zt + z * zz)):
        h = (n @ Z[0].T, -(n @ Z[1].T))
        h = (T[0].T @ h[0] + T[1].T @ h[1], T[0].T @ h[1] - T[1].T @ h[0])
        norm = L(1) / L(NTP * NZR)
        h = [x * norm for x in h]
        for x in h:
            x[NT // 2], x[:, NZ - 1] = 0, 0
        out.append(h)
    return out


def error(got, want, skip_mean):
    d = [got.real - want[0], got.imag - want[1]]
    w = [want[0].copy(), want[1].copy()]
    if skip_mean:
        for x in d + w:
            x[0, 0] = 0
    return float(np.sqrt(sum((x * x).sum() for x in d) / sum((x * x).sum() for x in w)))


@pytest.mark.parametrize("NT,NZ,spread", [(16, 33, 0), (32, 65, 0), (36, 55, 0), (18, 109, 0), (8, 193, 0), (64, 17, 0),
                                          (32, 65, 60), (18, 109, 60)])
def test_error_of_the_nonlinear_term(nsp, NT, NZ, spread):
    """White lines, and lines whose coefficients spread over `spread` octaves."""
    u = rough_field(NT, NZ, 21)
    u = [a[:NR].copy() for a in u]
    u[0][:] = 0
    if spread:
        m = np.minimum(np.arange(NT), NT - np.arange(NT))
        fall = np.exp2(-spread * (m.reshape(-1, 1) / (NT / 2.0) + np.arange(NZ) / (NZ - 1.0)) / 2)
        u = [a * fall for a in u]
    st = nsp.Stepper(nsp.make_params(NR, NT, NZ, Re, 0.01, LZ), precision=nsp.NSP_FP64)
    got = nonlinear(st, u)
    r = L(st.grid(0)[0][LEVEL])
    want = reference([u[1][LEVEL], u[2][LEVEL]], r, NT, NZ)
    err = [error(got[c][LEVEL], want[c], c == 2) for c in range(3)]
    assert max(err) < 5e-16, err
    st.close()
