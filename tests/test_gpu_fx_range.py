"""The FP64 form's nonlinear term at the ends of FP64's range: a transform line's scale follows
its values from subnormal ones to those whose sums still fit.

The field has a mean axial velocity W(r) and a radial one at every mode, u_theta = 0, so that
N_r = -i k_z W u_r and nothing else above FP64's rounding (u_r d_r u_r is smaller by u_r / W)."""
import numpy as np
import pytest

from conftest import PI2
from test_gpu_fx_transforms import LZ, NR, Re, nonlinear, rough_field
from test_gpu_parity import nsp  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu

# W of order 2^kw, u_r of order 2^ku.  1e-13 of the norm is the gate of the other operator tests.
# At 2^-1030 FP64's own unit, 2^-1074, is 6e-14 of a value of u_r: ten such roundings stay below 1e-12.
ENDS = [(1003, -500, 1e-13), (1003, -1000, 1e-13), (0, -890, 1e-13), (0, -930, 1e-13), (0, -960, 1e-13),
        (0, -1000, 1e-13), (0, -1030, 1e-12)]


def scale(a, k):
    return np.ldexp(np.ascontiguousarray(a).view(np.float64), k).view(np.complex128)


@pytest.mark.parametrize("NT,NZ", [(32, 65), (18, 109)])  # compiled and run-time lengths
@pytest.mark.parametrize("kw,ku,tol", ENDS)
def test_ends_of_the_range(nsp, NT, NZ, kw, ku, tol):
    st = nsp.Stepper(nsp.make_params(NR, NT, NZ, Re, 0.01, LZ), precision=nsp.NSP_FP64)
    r = st.grid(0)[0]
    u = rough_field(NT, NZ, 5)
    u[0][:, 0, 0] = 0
    u[0] = scale(u[0], ku)
    u[1][:], u[2][:] = 0, 0
    u[2][:, 0, 0] = np.ldexp(1.5 - r * r, kw)
    got = nonlinear(st, u)
    assert all(np.isfinite(a.view(np.float64)).all() for a in got)
    kz = np.arange(NZ) * (PI2 / LZ)
    want = -1j * kz * (1.5 - r * r).reshape(-1, 1, 1) * scale(u[0], -ku)
    assert np.linalg.norm(scale(got[0], -kw - ku) - want) < tol * np.linalg.norm(want)
    st.close()
