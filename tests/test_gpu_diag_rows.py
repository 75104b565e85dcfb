"""The divergence diagnostic at radial sizes around its split into blocks of 12 rows, each row
in turn carrying the maximum, against the CPU oracle.

Tolerance: a value is a sum of some 12 products, each good to a few ulp, and its terms add up to
at most ~100 times the maximum taken: 12 x 100 x 1e-16, with the stencil weights' own rounding
1e-12 relative."""
import numpy as np
import pytest

from conftest import PI2
from test_gpu_parity import nsp  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("NR", [8, 11, 12, 13, 24, 25, 31])
def test_divergence_maxima(nsp, oracle_lib, NR):
    NT, NZ, Re, LZ = 6, 7, 1500.0, 2 * PI2
    o = oracle_lib.Oracle(NR, NT, NZ, Re=Re, dt=0.01, LZ=LZ)
    st = nsp.Stepper([nsp.make_params(NR, NT, NZ, Re, 0.01, LZ)] * 2, precision=nsp.NSP_FP64)
    rng = np.random.default_rng(NR)
    base = [rng.standard_normal((NR, NT, NZ)) + 1j * rng.standard_normal((NR, NT, NZ)) for _ in range(3)]
    st.set_state(1, base)
    for i in range(NR):
        u = [a.copy() for a in base]
        for a in u:
            a[i] *= 1e3
        st.set_state(0, u)
        d = st.diag(0)
        ref, wall = np.abs(o.divergence(*u)[: NR - 1]).max(), np.abs(o.div_wall(*u)).max()
        assert abs(d.div_max - ref) <= 1e-12 * ref, i
        assert abs(d.div_wall - wall) <= 1e-12 * wall, i
    both = st.diag_all()
    assert (both[0].div_max, both[0].div_wall) == (d.div_max, d.div_wall)
    assert both[1].div_max == st.diag(1).div_max and both[1].div_wall == st.diag(1).div_wall
    st.close()
    o.close()
