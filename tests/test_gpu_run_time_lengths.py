"""Transform lengths without a compiled kernel (the run-time plan along theta, along z or both):
the nonlinear term and steps against the oracle, with the gates of the compiled lengths -- FP64
1e-13 for the term and 1e-12 with identical iteration counts after 10 steps, mixed 2e-6 and 1e-6 --
and the cross sections against the plain sums.  The shapes are checked to have no compiled transform."""
import os
import re

import numpy as np
import pytest

from conftest import PI2, ROOT, rel
from test_gpu_parity import dev, nsp  # noqa: F401  (fixture)

NR, Re, dt, LZ = 24, 1500.0, 0.005, PI2
# (NT, NZ): 27 x 324, 81 x 18, 27 x 12, 9 x 324, 81 x 96 and 24 x 324 points
SHAPES = [(18, 109), (54, 7), (18, 5), (6, 109), (54, 33), (16, 109)]


def compiled(which):
    with open(os.path.join(ROOT, "nspipe-gpu_gb300", "csrc", "nsp_fft.cuh")) as f:
        text = f.read().replace("\\\n", " ")
    line = re.search(r"#define NSP_%s_LIST\(X\)(.*)" % which, text).group(1)
    return {int(n) for n in re.findall(r"X\((\d+)\)", line)}


def test_shapes_are_run_time_ones():
    t, z = compiled("NTP"), compiled("NZR")
    assert t and z
    both = [(3 * NT // 2 not in t, 3 * (NZ - 1) not in z) for NT, NZ in SHAPES]
    assert all(a or b for a, b in both) and (True, True) in both and (True, False) in both and (False, True) in both


def stepper(nsp, NT, NZ, precision):
    st = nsp.Stepper(nsp.make_params(NR, NT, NZ, Re, dt, LZ), precision=precision)
    name = st.describe()["groups"][0]["z_stage"]
    assert name.startswith("radix") == (3 * (NZ - 1) not in compiled("NZR")), name
    return st


@pytest.mark.gpu
@pytest.mark.parametrize("NT,NZ", SHAPES)
def test_nonlinear_and_steps(nsp, oracle_lib, NT, NZ):
    import torch
    o = oracle_lib.Oracle(NR, NT, NZ, Re=Re, dt=dt, LZ=LZ)
    u0 = nsp.seeded_field(NR, NT, NZ, LZ, 0.02, 31)
    ref = o.nonlinear([a.copy() for a in u0])
    uo, ito, _ = o.step([a.copy() for a in u0], 10)
    o.close()
    for precision, tol_n, tol_u in ((nsp.NSP_FP64, 1e-13, 1e-12), (nsp.NSP_MIXED, 2e-6, 1e-6)):
        st = stepper(nsp, NT, NZ, precision)
        n = [torch.zeros(u0[0].shape, dtype=torch.complex128, device="cuda") for _ in range(3)]
        st.nonlinear(0, [dev(a) for a in u0], n)
        for c in range(3):
            assert rel(n[c].cpu().numpy(), ref[c]) < tol_n, (precision, c)
        st.set_state(0, u0)
        it = st.step(10)
        if precision == nsp.NSP_FP64:
            assert list(it[:, 0]) == list(ito)
        assert rel(np.stack(st.get_state(0)), np.stack(uo)) < tol_u, precision
        st.close()


@pytest.mark.gpu
@pytest.mark.parametrize("NT,NZ", SHAPES)
def test_cross_sections(nsp, NT, NZ):
    u = nsp.seeded_field(NR, NT, NZ, LZ, 0.02, 32)
    st = stepper(nsp, NT, NZ, nsp.NSP_MIXED)
    st.set_state(0, u)
    q, w = st.cross_sections(0)
    rdr, nzr = st.grid(0)[1], 3 * (NZ - 1)
    st.close()
    e = np.exp(2j * np.pi * (np.outer(np.arange(NZ), np.arange(nzr)) % nzr) / nzr)
    ms = []
    for a in u:
        p = 2.0 * (a[:, :, 1:] @ e[1:]) + a[:, :, :1]
        s = p[:, 0].real ** 2 + 0.5 * np.abs(p[:, NT // 2]) ** 2
        for mu in range(1, NT // 2):
            s = s + 2.0 * np.abs(0.5 * (p[:, mu] + p[:, NT - mu].conj())) ** 2
        ms.append(rdr @ s)
    assert rel(q, ms[0] + ms[1]) < 1e-13 and rel(w, ms[2]) < 1e-13
