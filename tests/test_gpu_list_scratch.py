"""Which states take the scratch of the list forms, by the bytes in use in the device's
memory pool."""
import ctypes as C

import numpy as np
import pytest

import cases as K

pytestmark = pytest.mark.gpu

S = pytest.importorskip("sphadjoint_gb300")
PAIRS = 1290  # bytes a particle of the FP64 pair lists


def pool():
    L = C.CDLL("libcuda.so.1")
    dev, p = C.c_int(), C.c_void_p()
    assert L.cuDeviceGet(C.byref(dev), 0) == 0
    assert L.cuDeviceGetDefaultMemPool(C.byref(p), dev) == 0
    return L, p


def used():
    """Bytes in use (CU_MEMPOOL_ATTR_USED_MEM_CURRENT) after all frees have run."""
    L, p = pool()
    S.synchronize()
    v = C.c_uint64()
    assert L.cuMemPoolGetAttribute(p, 7, C.byref(v)) == 0
    return v.value


def state(nx, ny, dtype="f64", **model):
    dx = 0.01
    p = K.dambreak_params(dx=dx, col_h=ny * dx, Lx=2.0 * nx * dx, Ly=1.25 * max(nx, ny) * dx)
    p.update(model)
    rng = np.random.default_rng(nx + ny)
    X0 = K.lattice_block(nx, ny, dx, dx, dx, 0.05 * dx, rng)
    sp = S.SPHParams(**p, dtype=dtype)
    th = S.DesignField(20.0 * rng.random((p["ngy"], p["ngx"])), dtype)
    return S.State(X0, 0.2 * rng.standard_normal(X0.shape), sp, interval=2), th, sp


@pytest.mark.parametrize("model,takes", [({}, True), (dict(visc=1, alpha=0.02), False)])
def test_only_models_with_pair_passes_take_pair_lists(model, takes):
    st, th, sp = state(80, 60, **model)
    before = used()
    S.step(st, th)
    assert (used() - before >= PAIRS * st.N) == takes
    if not takes:  # the same state with a model that has them
        sp.visc = "morris" if isinstance(sp.visc, str) else 0
        S.step(st, th, sp)
        assert used() - before >= PAIRS * st.N


@pytest.mark.parametrize("dtype,nx,ny", [("f64", 700, 700), ("f32", 2000, 1600)])
def test_refused_lists_are_asked_for_again(dtype, nx, ny):
    """Lists are taken from an eighth of the free memory at most. A state that starts while
    less is free steps without them, and takes them once there is room; its results are
    those of a state that had them from the start."""
    torch = pytest.importorskip("torch")
    ref, th, _ = state(nx, ny, dtype)
    st, _, _ = state(nx, ny, dtype)
    least = (PAIRS if dtype == "f64" else 195) * st.N
    before = used()
    S.step(ref, th)
    assert used() - before >= least
    L, p = pool()
    assert L.cuMemPoolTrimTo(p, C.c_size_t(0)) == 0
    hog = torch.empty(torch.cuda.mem_get_info()[0] - 5 * least, dtype=torch.uint8, device="cuda")
    before = used()
    S.step(st, th)
    assert used() == before  # refused
    del hog
    torch.cuda.empty_cache()
    for _ in range(2):
        S.step(st, th)
    assert used() - before >= least
    for _ in range(2):
        S.step(ref, th)
    for a, b in zip(st.get(), ref.get()):
        assert np.array_equal(a, b)
