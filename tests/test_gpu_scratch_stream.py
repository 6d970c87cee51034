"""The lists of a state are taken at its first step, on whatever stream the caller has set by
then. They are given back with the state's other buffers, so that stream may be destroyed
before the state."""
import ctypes as C

import numpy as np
import pytest

import cases as K

pytestmark = pytest.mark.gpu

S = pytest.importorskip("sphadjoint_gb300")
from sphadjoint_gb300 import _lib as LB  # noqa: E402


def used(cu):
    """Bytes in use in the device's memory pool (CU_MEMPOOL_ATTR_USED_MEM_CURRENT)."""
    dev, pool, v = C.c_int(), C.c_void_p(), C.c_uint64()
    S.synchronize()
    assert cu.cuDeviceGet(C.byref(dev), 0) == 0
    assert cu.cuDeviceGetDefaultMemPool(C.byref(pool), dev) == 0
    assert cu.cuMemPoolGetAttribute(pool, 7, C.byref(v)) == 0
    return v.value


@pytest.mark.parametrize("dtype,nx,ny,least", [("f32", 150, 120, 195), ("f64", 60, 50, 1290)])
def test_stream_of_the_first_step_destroyed_before_the_state(dtype, nx, ny, least):
    dx = 0.01
    p = K.dambreak_params(dx=dx, col_h=ny * dx, Lx=2.0 * nx * dx, Ly=1.25 * max(nx, ny) * dx)
    X0 = K.lattice_block(nx, ny, dx, dx, dx, 0.05 * dx, np.random.default_rng(nx))
    sp = S.SPHParams(**p, dtype=dtype)
    th = S.DesignField(np.zeros((p["ngy"], p["ngx"])), dtype)
    cu = C.CDLL("libcuda.so.1")
    before = used(cu)
    st = S.State(X0, np.zeros_like(X0), sp, interval=2)
    ref = S.State(X0, np.zeros_like(X0), sp, interval=2)
    S.synchronize()
    own = used(cu)
    stream = C.c_void_p()
    assert cu.cuStreamCreate(C.byref(stream), 1) == 0
    LB.check(S.load().sph_set_stream(stream))
    try:
        S.step(st, th)
        S.synchronize()
    finally:
        LB.check(S.load().sph_set_stream(None))
        assert cu.cuStreamDestroy_v2(stream) == 0
    assert used(cu) - own >= least * st.N
    for _ in range(2):  # and the state goes on
        S.step(st, th)
    for _ in range(3):
        S.step(ref, th)
    for a, b in zip(st.get(), ref.get()):
        assert np.array_equal(a, b)
    del st, ref
    assert used(cu) == before
