"""Cell lists whose tables end at, just before and just after the tiles of their
scan, and beyond the number of tiles that a block sums itself: counts, starts and
order bit for bit against the oracle, also from a second and third list of the same
state (the counters have to be zero again after each)."""
import numpy as np
import pytest

import cases as K

pytestmark = pytest.mark.gpu

S = pytest.importorskip("sphadjoint_gb300")
import oracle as O  # noqa: E402

# nx, ny: 2047, 2048 and 2049 cells (tiles of 2048), two tiles and a cell, 4096
# tiles, 4102 tiles
GRIDS = [(89, 23), (64, 32), (683, 3), (17, 241), (2048, 4096), (3000, 2800)]


@pytest.mark.parametrize("nx,ny", GRIDS)
@pytest.mark.parametrize("n", [4097, 6151])
def test_cell_list_at_the_tiles_of_the_scan(nx, ny, n):
    p = dict(K.dambreak_params())
    cs = 2.0 * p["h"] * 1.2
    p["Lx"], p["Ly"] = (nx - 2.5) * cs, (ny - 2.5) * cs
    rng = np.random.default_rng(n + nx)
    X = rng.random((2, n)) * np.array([[p["Lx"]], [p["Ly"]]])
    X[:, :40] = [[1e6], [1e6]]      # the table's last cell
    X[:, 40:90] = [[-1e6], [-1e6]]  # and its first
    X[:, 90:2000] *= 0.02           # crowded cells, most of one warp in one
    st = S.State(X, np.zeros_like(X), S.SPHParams(**p))
    ost = O.Oracle("f64").state(O.params(**p), X, np.zeros_like(X))
    ost.build_cells()
    want = ost.cells()
    assert want["counts"].size == nx * ny
    for build in (S.build, S.build, S.build_neighbors, S.build):
        build(st)
        got = st.celllist()
        for key in ("counts", "starts", "order"):
            assert np.array_equal(got[key], want[key]), (key, build.__name__)
