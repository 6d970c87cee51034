"""Neighbour lists made inside a recording exist only once it is replayed, and those made
outside may be of other masks when it is. So a recording of FP32 tile steps makes the lists
it needs from the masks it finds: replayed again from an earlier state it gives the same
bits, and a recording that is dropped leaves the state as it was."""
import numpy as np
import pytest

import cases as K

pytestmark = pytest.mark.gpu

S = pytest.importorskip("sphadjoint_gb300")


def states():
    dx, nx, ny = 0.01, 150, 120
    p = K.dambreak_params(dx=dx, col_h=ny * dx, Lx=2.0 * nx * dx, Ly=1.25 * nx * dx)
    rng = np.random.default_rng(5)
    X0 = K.lattice_block(nx, ny, dx, dx, dx, 0.05 * dx, rng)
    sp = S.SPHParams(**p, dtype="f32")
    th = S.DesignField(20.0 * rng.random((p["ngy"], p["ngx"])), "f32")
    V0 = 2.0 * rng.standard_normal(X0.shape)
    new = lambda: S.State(X0, V0, sp, interval=4)  # noqa: E731
    st, kept, ref = new(), new(), new()
    for _ in range(2):  # within a rebuild interval
        S.step(st, th)
        S.step(ref, th)
    kept.assign(st)
    return st, kept, ref, th


def steps(st, th, n):
    for _ in range(n):
        S.step(st, th)


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a.get(), b.get()))


def test_replay_from_an_earlier_state():
    st, kept, ref, th = states()
    # two steps on the old list, a rebuild, three on the new: the buffers end as they began
    g = S.capture(lambda: steps(st, th, 5))
    steps(ref, th, 5)
    for _ in range(3):
        st.assign(kept)
        g.launch()
        S.synchronize()
        assert same(st, ref)


def test_dropped_recording():
    st, kept, ref, th = states()
    st.assign(kept)  # masks without lists
    g = S.capture(lambda: steps(st, th, 5))
    del g
    steps(st, th, 1)
    steps(ref, th, 1)
    assert same(st, ref)
