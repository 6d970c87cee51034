"""FP64 cell lists whose coordinates sit on and around cell borders: the float
estimate of x / cs must leave those to the division (counts, starts and order
bit for bit against the oracle), in the one-launch cell list of small states and
in the multi-launch one."""
import numpy as np
import pytest

import cases as K

pytestmark = pytest.mark.gpu

S = pytest.importorskip("sphadjoint_gb300")
import oracle as O  # noqa: E402


@pytest.mark.parametrize("n", [700, 9000])
@pytest.mark.parametrize("rebuild", [False, True])
def test_cells_on_borders(n, rebuild):
    rng = np.random.default_rng(n)
    p = K.dambreak_params()
    cs = 2.0 * p["h"] * 1.2
    k = rng.integers(-2, int(p["Lx"] / cs) + 3, size=(2, n))
    ulps = rng.integers(-3, 4, size=(2, n))
    X = k * cs
    X = X + ulps * np.spacing(np.abs(X) + 1e-300)
    X[:, ::7] = rng.random(X[:, ::7].shape) * p["Lx"]
    X[0, :5] = [0.0, -0.0, 1e-310, -1e-310, 5e5]
    st = S.State(X, np.zeros_like(X), S.SPHParams(**p))
    ost = O.Oracle("f64").state(O.params(**p), X, np.zeros_like(X))
    if rebuild:
        S.build_neighbors(st)
        ost.build_neighbors(p["h"])
    else:
        S.build(st)
        ost.build_cells()
    g, c = st.celllist(), ost.cells()
    for key in ("counts", "starts", "order"):
        assert np.array_equal(g[key], c[key]), key


@pytest.mark.parametrize("lanes", [1, 16, 32])
def test_neighbour_rows_at_the_cutoff(lanes):
    """Pairs whose distance is the list's cutoff up to a few ulps, coincident
    particles, particles far outside the tank (clamped into border cells) and tiny
    offsets: the float estimate of r^2 must leave those to the FP64 test. Rows and
    counts as the oracle lists them."""
    rng = np.random.default_rng(5)
    p = K.dambreak_params()
    rc = 2.0 * p["h"] * 1.2
    n = 600
    X = np.empty((2, n))
    X[:, 0::3] = np.vstack([0.1 + 1.4 * rng.random(n // 3), 0.1 + 0.8 * rng.random(n // 3)])
    a = rng.choice([0.0, 0.5 * np.pi, np.pi, 1.0, 2.5], n // 3)
    d = rc * (1.0 + rng.integers(-3, 4, n // 3) * 2.0 ** -52)
    X[:, 1::3] = X[:, 0::3] + d * np.vstack([np.cos(a), np.sin(a)])
    X[:, 2::3] = X[:, 0::3]                       # coincident with the first
    X[0, 2::6] += p["h"] * 2.0 ** -26             # or at r^2 about eps h^2
    X[:, 5::60] = 1e3 * (1.0 + rng.random(X[:, 5::60].shape))
    X[:, 8::60] = -0.2 * rng.random(X[:, 8::60].shape)
    try:
        S.set_group_lanes(lanes)
        st = S.State(X, np.zeros_like(X), S.SPHParams(**p))
        S.build_neighbors(st)
        gi, gn = st.neighbors()
    finally:
        S.set_group_lanes(0)
    ost = O.Oracle("f64").state(O.params(**p), X, np.zeros_like(X))
    ost.build_neighbors(p["h"])
    oi, on = ost.neighbors()
    assert np.array_equal(gn, on)
    for i in range(n):
        assert np.array_equal(gi[i, : gn[i]], oi[i, : on[i]]), i
