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
