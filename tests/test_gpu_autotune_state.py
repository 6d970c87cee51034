"""Tuning block sizes leaves the state as it was: in the middle of a rebuild interval, with
particles that have moved since the neighbours were listed, the rows, the flags and the
steps that follow equal those of a state that was not tuned, whether it holds lists or not."""
import ctypes as C

import numpy as np
import pytest

import cases as K

pytestmark = pytest.mark.gpu

S = pytest.importorskip("sphadjoint_gb300")


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("form", ["pairs", "mask"])
def test_tuning_within_a_rebuild_interval(dtype, form):
    dx, nx, ny = 0.01, 150, 120
    p = K.dambreak_params(dx=dx, col_h=ny * dx, Lx=2.0 * nx * dx, Ly=1.25 * nx * dx)
    rng = np.random.default_rng(3)
    X0 = K.lattice_block(nx, ny, dx, dx, dx, 0.05 * dx, rng)
    # fast enough for pairs to cross the list's cutoff within a few steps
    V0 = 0.02 * p["h"] / p["dt"] * rng.standard_normal(X0.shape)
    sp = S.SPHParams(**p, dtype=dtype)
    th = S.DesignField(np.zeros((p["ngy"], p["ngx"])), dtype)
    tuned, other = (S.State(X0, V0, sp, interval=6) for _ in range(2))
    sizes = tuned.block_sizes()
    S.set_density_form(form)
    try:
        for st in (tuned, other):
            for _ in range(3):
                S.step(st, th)
        b6 = (C.c_int32 * 6)()
        assert S.load().sph_autotune(tuned.h, th.h, 1, b6) == 0
        tuned.set_block_sizes(sizes)
        (ai, an), (bi, bn) = tuned.neighbors(), other.neighbors()
        assert np.array_equal(an, bn) and np.array_equal(ai, bi)
        for st in (tuned, other):
            for _ in range(2):
                S.step(st, th)
        for a, b in zip(tuned.get(), other.get()):
            assert np.array_equal(a, b)
        assert tuned.take_flags() == other.take_flags()
    finally:
        S.set_density_form("pairs")
        tuned.set_block_sizes(sizes)
