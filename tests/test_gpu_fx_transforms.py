"""The FP64 form's transforms (64-bit fixed point inside, one scale per transform line)
against the CPU oracle's FP64 ones: every compiled length and run-time ones, in both
directions, and the scale of the lines over FP64's range.

Tolerance: the oracle's own transforms are within 5e-16 of the exact ones and a line's
fixed-point unit is 2^-61 of its sum of magnitudes, below FP64's rounding; the radial
derivative (7 terms, weights up to ~1/h at the wall) and the products carry a few ulp each.
1e-13 of the norm, the gate of the other operator tests, is some 100 times that."""
import numpy as np
import pytest

from conftest import PI2, rel
from test_gpu_parity import dev, nsp  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu

# (NT, NZ): theta lengths 3 NT / 2 and z lengths 3 (NZ - 1)
SHAPES = [(8, 9), (16, 17), (32, 33), (48, 65), (64, 129), (96, 193), (128, 257),  # 12..192 x 24..768
          (4, 3), (6, 5), (12, 13), (24, 25), (36, 55), (72, 19), (18, 49), (54, 97), (16, 145), (32, 37), (8, 73), (4, 109)]
NR, Re, LZ = 9, 1500.0, 2 * PI2


def nonlinear(st, u):
    import torch
    n = [torch.zeros(u[0].shape, dtype=torch.complex128, device="cuda") for _ in range(3)]
    st.nonlinear(0, [dev(a) for a in u], n)
    return [a.cpu().numpy() for a in n]


def rough_field(NT, NZ, seed):
    """Every retained mode of order 1 with the k_z = 0 plane of a real field: white lines."""
    rng = np.random.default_rng(seed)
    u = [rng.standard_normal((NR, NT, NZ)) + 1j * rng.standard_normal((NR, NT, NZ)) for _ in range(3)]
    for a in u:
        a[:, NT // 2], a[:, :, NZ - 1] = 0, 0
        a[:, 0, 0] = a[:, 0, 0].real
        for t in range(1, NT // 2):
            a[:, NT - t, 0] = a[:, t, 0].conj()
    return u


@pytest.mark.parametrize("NT,NZ", SHAPES)
def test_nonlinear_lengths(nsp, oracle_lib, NT, NZ):
    o = oracle_lib.Oracle(NR, NT, NZ, Re=Re, dt=0.01, LZ=LZ)
    st = nsp.Stepper(nsp.make_params(NR, NT, NZ, Re, 0.01, LZ), precision=nsp.NSP_FP64)
    for u in (rough_field(NT, NZ, 7), nsp.seeded_field(NR, NT, NZ, LZ, 1e-3, 8)):
        got, ref = nonlinear(st, u), o.nonlinear([a.copy() for a in u])
        for c in range(3):
            assert rel(got[c], ref[c]) < 1e-13, c
    st.close()
    o.close()


@pytest.mark.parametrize("NT,NZ", SHAPES)
def test_nonlinear_lengths_mixed(nsp, oracle_lib, NT, NZ):
    """The mixed form's FP32 transforms over the same lengths: a transform of n points leaves
    about 6e-8 log2(n) of its norm, three in a row with the products 2e-6 (the operator gate)."""
    o = oracle_lib.Oracle(NR, NT, NZ, Re=Re, dt=0.01, LZ=LZ)
    st = nsp.Stepper(nsp.make_params(NR, NT, NZ, Re, 0.01, LZ), precision=nsp.NSP_MIXED)
    u = rough_field(NT, NZ, 7)
    got, ref = nonlinear(st, u), o.nonlinear([a.copy() for a in u])
    for c in range(3):
        assert rel(got[c], ref[c]) < 2e-6, c
    st.close()
    o.close()


@pytest.mark.parametrize("NT,NZ", SHAPES)
def test_cross_sections_lengths(nsp, NT, NZ):
    """q and u as the theta means of the squared physical fields (numpy transforms).  Both sum
    squares of transforms good to 1e-15 of their norm: 1e-13 relative."""
    st = nsp.Stepper(nsp.make_params(NR, NT, NZ, Re, 0.01, LZ), precision=nsp.NSP_FP64)
    u = rough_field(NT, NZ, 11)
    rng = np.random.default_rng(12)
    for a in u:  # the slots without a partner count too
        a[:, NT // 2] = rng.standard_normal((NR, NZ)) + 1j * rng.standard_normal((NR, NZ))
        a[:, :, NZ - 1] = rng.standard_normal((NR, NT))
    st.set_state(0, u)
    q, w = st.cross_sections(0)
    rdr = st.grid(0)[1]
    nzr = 3 * (NZ - 1)
    e = np.exp(2j * np.pi * np.outer(np.arange(NZ), np.arange(nzr)) / nzr)
    ms = []
    for a in u:
        p = 2.0 * (a[:, :, 1:] @ e[1:]) + a[:, :, :1]
        s = p[:, 0].real ** 2 + 0.5 * np.abs(p[:, NT // 2]) ** 2
        for mu in range(1, NT // 2):
            s = s + 2.0 * np.abs(0.5 * (p[:, mu] + p[:, NT - mu].conj())) ** 2
        ms.append(rdr @ s)
    assert rel(q, ms[0] + ms[1]) < 1e-13 and rel(w, ms[2]) < 1e-13
    qa, wa = st.cross_sections_all()
    assert np.array_equal(qa[0], q) and np.array_equal(wa[0], w)
    st.close()


@pytest.mark.parametrize("NT,NZ", [(32, 65), (12, 13)])
def test_scale(nsp, NT, NZ):
    """N is quadratic in u, so a power of two comes out exactly, but for the wall forcing of
    the mean axial mode (linear in u): each line's scale follows its values."""
    st = nsp.Stepper(nsp.make_params(NR, NT, NZ, Re, 0.01, LZ), precision=nsp.NSP_FP64)
    u = rough_field(NT, NZ, 9)
    base = nonlinear(st, u)
    for k in (-400, -30, 30, 400):
        got = nonlinear(st, [np.ldexp(a.view(np.float64), k).view(np.complex128) for a in u])
        for c in range(3):
            g, b = got[c].copy(), base[c].copy()
            if c == 2:
                g[:, 0, 0], b[:, 0, 0] = 0, 0
            assert np.array_equal(g, np.ldexp(b.view(np.float64), 2 * k).view(np.complex128)), (k, c)
    z = nonlinear(st, [np.zeros_like(a) for a in u])
    assert all(not a.any() for a in z)
    st.close()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_line(nsp, bad):
    """One Inf or NaN coefficient makes N non-finite at its level and leaves others alone."""
    NT, NZ = 32, 65
    st = nsp.Stepper(nsp.make_params(24, NT, NZ, Re, 0.01, LZ), precision=nsp.NSP_FP64)
    u = nsp.seeded_field(24, NT, NZ, LZ, 1e-2, 3)
    good = nonlinear(st, u)
    u[0][20, 3, 2] = bad
    got = nonlinear(st, u)
    assert not np.isfinite(got[0][20].view(np.float64)).all()
    for c in range(3):
        assert np.array_equal(got[c][:17], good[c][:17])  # out of reach of the 7-point derivative
    st.close()
