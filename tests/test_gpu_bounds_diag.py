"""The bounds-checked build over what is called between the steps: device hand-over, the
diagnostics and the cross sections, one member and all of them, and steps at transform lengths
that have no compiled kernel.  No violation is recorded, and the values are the normal build's."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import PI2, ROOT
from test_gpu_parity import nsp  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu

# NR, NT, NZ: run-time lengths (27 x 324, 81 x 18, 9 x 324), compiled ones, edges of the rows' blocks
SHAPES = [(24, 18, 109), (13, 54, 7), (8, 6, 109), (8, 4, 3), (25, 8, 9), (12, 16, 17), (48, 32, 65)]

BODY = r'''
def collect(nsp, shapes, PI2):
    import numpy as np
    import torch
    out, bounds = [], []
    for prec in (nsp.NSP_FP64, nsp.NSP_MIXED):
        for k, s in enumerate(shapes):
            prm = [nsp.make_params(*s, 1000.0 + 100 * j, 0.005, PI2) for j in range(3)]
            prm.append(nsp.make_params(16, 12, 13, 900.0, 0.005, PI2))  # a second group
            st = nsp.Stepper(prm, precision=prec)
            for m, p in enumerate(prm):
                u = nsp.seeded_field(p.NR, p.NT, p.NZ, p.LZ, 0.02, 40 + 7 * k + m)
                st.set_state_device(m, *[torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in u])
            st.step(2)
            for m, p in enumerate(prm):
                u = [torch.zeros((p.NR, p.NT, p.NZ), dtype=torch.complex128, device="cuda") for _ in range(3)]
                torch.cuda.synchronize()
                st.get_state_device(m, *u)
                out += [a.cpu().numpy().reshape(-1).view(np.float64) for a in u]
                out += list(st.cross_sections(m)) + [st.mean_profile(m)]
                d = st.diag(m)
                out.append(np.array([d.u_centre, d.u_tau, d.flux, d.re_tau]))
            q, w = st.cross_sections_all()
            out += list(q) + list(w) + list(st.mean_profile_all())
            out += [np.array([d.div_max, d.div_wall]) for d in st.diag_all()]
            bounds.append(list(st.bounds_report()))
            st.close()
    return out, bounds
'''
CHILD = BODY + r'''
import sys
import numpy as np
import nspipe_gb300 as nsp
assert nsp.LIB_PATH.endswith("_bc.so"), nsp.LIB_PATH
out, bounds = collect(nsp, eval(sys.argv[2]), nsp.PI2)
np.savez(sys.argv[1], bounds=np.array(bounds), **{"a%d" % k: a for k, a in enumerate(out)})
'''


def test_checked_build_between_steps(nsp, tmp_path):
    import build as nbuild
    lib = nbuild.build(bounds_check=True)
    f = str(tmp_path / "out.npz")
    env = dict(os.environ, NSP_LIBRARY=lib, PYTHONPATH=os.path.join(ROOT, "nspipe-gpu_gb300"))
    p = subprocess.run([sys.executable, "-c", CHILD, f, repr(SHAPES)], env=env, capture_output=True, text=True, timeout=900)
    assert p.returncode == 0, p.stdout[-3000:] + p.stderr[-3000:]
    got = np.load(f)
    for b in got["bounds"]:
        assert b[4] == 1 and b[0] == 0, list(b)  # the checked build; (count, site, index, extent)
    scope = {}
    exec(BODY, scope)
    want, _ = scope["collect"](nsp, SHAPES, PI2)
    assert len(want) == len(got.files) - 1
    for k, a in enumerate(want):
        # values of order 1 by the same operations in the same order: FP64's rounding where the compiler contracts them
        # differently, FP32's after two steps of the mixed form
        tol = 1e-12 if k < len(want) // 2 else 1e-6
        assert np.linalg.norm(got["a%d" % k] - a) <= tol * max(np.linalg.norm(a), 1.0), (k, a.size)
