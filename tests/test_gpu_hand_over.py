"""State hand-over between device arrays (nsp_set_state_device / nsp_get_state_device): the
values arrive bit for bit whatever the arrays are -- aligned or on an 8-byte boundary, apart,
side by side, the last of an allocation, managed memory, written on a stream of the caller's --
and where the destinations of a get overlap, as three copies in the order u_r, u_theta, u_z."""
import ctypes

import numpy as np
import pytest

from conftest import PI2
from test_gpu_parity import nsp  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu

SHAPES = [(8, 4, 3), (24, 8, 9), (61, 36, 55)]  # 96, 1728 and 120780 values; copy blocks hold 1024


def stepper(nsp, shape, n=2):
    return nsp.Stepper([nsp.make_params(*shape, 1200.0, 0.005, PI2)] * n, precision=nsp.NSP_FP64)


def fields(shape, seed):
    rng = np.random.default_rng(seed)
    return [rng.standard_normal(shape) + 1j * rng.standard_normal(shape) for _ in range(3)]


def words(n, offset=0):
    """A float64 tensor of 6 n + 16 values and its start; offset in 8-byte words."""
    import torch
    t = torch.full((6 * n + 16,), -7.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    return t, t.data_ptr() + 8 * offset


def bits(a):
    return np.ascontiguousarray(a).reshape(-1).view(np.float64)


# starts of the three arrays in 8-byte words, n complex values each
APART = {"side by side": lambda n: (0, 2 * n, 4 * n), "8 bytes off": lambda n: (1, 2 * n + 1, 4 * n + 1),
         "one off": lambda n: (0, 2 * n + 1, 4 * n + 2), "gaps, any order": lambda n: (4 * n + 8, 0, 2 * n + 4)}


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("layout", sorted(APART))
def test_round_trip(nsp, shape, layout):
    import torch
    n = int(np.prod(shape))
    at = APART[layout](n)
    st = stepper(nsp, shape)
    u, other = fields(shape, 1), fields(shape, 2)
    st.set_state(0, other)
    src, _ = words(n)
    for k in range(3):
        src[at[k]: at[k] + 2 * n] = torch.from_numpy(bits(u[k]))
    torch.cuda.synchronize()
    st.set_state_device(1, *[src.data_ptr() + 8 * a for a in at])
    for k in range(3):
        assert np.array_equal(st.get_state(1)[k], u[k]) and np.array_equal(st.get_state(0)[k], other[k])
    dst, p = words(n)
    st.get_state_device(1, *[p + 8 * a for a in at])
    assert torch.equal(dst, src)  # the values, and nothing beside them
    st.close()


# destinations that share memory: what three copies in order leave
SHARED = {"all one": lambda n: (0, 0, 0), "first and last": lambda n: (0, 2 * n, 0), "first two": lambda n: (0, 0, 2 * n),
          "last two": lambda n: (2 * n, 0, 0), "half": lambda n: (0, n - n % 2, 2 * (n - n % 2)),
          "half, backwards": lambda n: (2 * (n - n % 2), n - n % 2, 0),
          "one value": lambda n: (0, 2 * n - 2, 4 * n - 4), "one word": lambda n: (0, 2 * n - 1, 4 * n - 2)}


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("layout", sorted(SHARED))
def test_overlapping_arrays(nsp, shape, layout):
    import torch
    n = int(np.prod(shape))
    at = SHARED[layout](n)
    st = stepper(nsp, shape, 1)
    u = fields(shape, 3)
    st.set_state(0, u)
    dst, p = words(n)
    want = dst.cpu().numpy()
    for k in range(3):
        want[at[k]: at[k] + 2 * n] = bits(u[k])
    for _ in range(3):
        st.get_state_device(0, *[p + 8 * a for a in at])
        assert np.array_equal(dst.cpu().numpy(), want)
    # a set reads them: each component is what lies there
    st.set_state_device(0, *[p + 8 * a for a in at])
    for k in range(3):
        assert np.array_equal(bits(st.get_state(0)[k]), want[at[k]: at[k] + 2 * n])
    torch.cuda.synchronize()
    st.close()


@pytest.mark.parametrize("managed", [False, True])
def test_whole_allocation(nsp, managed):
    """Arrays that fill an allocation of the driver's to its last byte, and managed memory."""
    import torch
    shape = SHAPES[1]
    n = int(np.prod(shape))
    st = stepper(nsp, shape, 1)
    torch.zeros(1, device="cuda")  # (the device's primary context is current)
    cu = ctypes.CDLL("libcuda.so.1")
    p = ctypes.c_uint64(0)
    size = ctypes.c_size_t(48 * n)
    rc = cu.cuMemAllocManaged(ctypes.byref(p), size, 1) if managed else cu.cuMemAlloc_v2(ctypes.byref(p), size)
    assert rc == 0
    u = fields(shape, 4)
    st.set_state(0, u)
    at = [p.value + 16 * n * k for k in range(3)]
    st.get_state_device(0, *at)
    st.set_state(0, fields(shape, 5))
    st.set_state_device(0, *at)
    for k in range(3):
        assert np.array_equal(st.get_state(0)[k], u[k])
    assert cu.cuMemFree_v2(p) == 0
    st.close()


def test_callers_stream(nsp):
    """On a stream of the caller's the hand-over follows the work queued there."""
    import torch
    shape = SHAPES[2]
    st = stepper(nsp, shape, 1)
    u = fields(shape, 6)
    stream = torch.cuda.Stream()
    st.set_stream(stream.cuda_stream)
    base = [torch.from_numpy(a).cuda() for a in u]
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        x = [a.clone() for a in base]
        for _ in range(50):
            x = [-a for a in x]
        st.set_state_device(0, *x)
        y = [torch.zeros_like(a) for a in x]
        st.get_state_device(0, *y)
        z = [2.0 * a for a in y]
    torch.cuda.synchronize()
    for k in range(3):
        assert np.array_equal(z[k].cpu().numpy(), 2.0 * u[k])
    st.set_stream(None)
    st.close()
