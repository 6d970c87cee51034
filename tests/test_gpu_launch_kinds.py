"""What each form launches for a step, by the library's kernel timers: the density pass of a
rebuild step that builds the masks too is timed apart from the density passes alone, and the
default forms are the ones that run (mask walks build the masks in a launch of their own)."""
import ctypes as C

import numpy as np
import pytest

import cases as K

pytestmark = pytest.mark.gpu

S = pytest.importorskip("sphadjoint_gb300")
from sphadjoint_gb300 import _lib as LB  # noqa: E402

NAMES = ("rank", "nl_build", "density", "build_density", "accel_integrate")


def counts(dtype, nx, ny, steps):
    dx = 0.01
    p = K.dambreak_params(dx=dx, col_h=ny * dx, Lx=2.0 * nx * dx, Ly=1.25 * max(nx, ny) * dx)
    rng = np.random.default_rng(nx)
    X0 = K.lattice_block(nx, ny, dx, dx, dx, 0.05 * dx, rng)
    sp = S.SPHParams(**p, dtype=dtype)
    th = S.DesignField(np.zeros((p["ngy"], p["ngx"])), dtype)
    st = S.State(X0, np.zeros_like(X0), sp, interval=3)
    L = S.load()
    LB.check(L.sph_profile_reset())
    try:
        for k in NAMES:
            LB.check(L.sph_profile_enable(LB.KERNEL_ID[k], 1))
        for _ in range(steps):
            S.step(st, th)
        out = {}
        for k in NAMES:
            ms, n = C.c_double(), C.c_int64()
            LB.check(L.sph_profile_read(LB.KERNEL_ID[k], C.byref(ms), C.byref(n)))
            out[k] = n.value
        return out
    finally:
        for k in NAMES:
            LB.check(L.sph_profile_enable(LB.KERNEL_ID[k], 0))
        LB.check(L.sph_profile_reset())


# tiles; lane groups; pairs with 4 particles a block; pairs with more than 8 a block
@pytest.mark.parametrize("dtype,nx,ny,fused", [("f32", 150, 120, True), ("f32", 40, 30, True),
                                               ("f64", 40, 30, True), ("f64", 80, 60, False)])
def test_default_forms(dtype, nx, ny, fused):
    c = counts(dtype, nx, ny, 7)  # rebuilds at steps 1, 4 and 7
    assert c["rank"] == 3 and c["accel_integrate"] == 7
    assert (c["nl_build"], c["build_density"], c["density"]) == ((0, 3, 4) if fused else (3, 0, 7))


def test_mask_walks():
    S.set_density_form("mask")
    try:
        c = counts("f32", 150, 120, 7)
    finally:
        S.set_density_form("pairs")
    assert (c["nl_build"], c["build_density"], c["density"]) == (3, 0, 7)
