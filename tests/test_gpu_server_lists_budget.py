"""The lists of a request's states are charged to the server's budget, and left out where it
has no room for them: a request whose estimate fits is still admitted, the admitted bytes
stay within the budget, and the results are the same bits."""
import numpy as np
import pytest

import cases as K

pytestmark = pytest.mark.gpu

S = pytest.importorskip("sphadjoint_gb300")
from sphadjoint_gb300.serve import Server  # noqa: E402


def request(nx, ny, dtype):
    dx = 0.01
    p = K.dambreak_params(dx=dx, col_h=ny * dx, Lx=2.0 * nx * dx, Ly=1.25 * max(nx, ny) * dx)
    rng = np.random.default_rng(nx + ny)
    X0 = K.lattice_block(nx, ny, dx, dx, dx, 0.05 * dx, rng)
    return (S.SPHParams(**p, dtype=dtype), X0, 0.2 * rng.standard_normal(X0.shape),
            20.0 * rng.random((p["ngy"], p["ngx"])))


def serve(req, packed, budget, count=1):
    p, X0, V0, th = req
    kw = dict(packed=True) if packed else dict(workers=2)
    n0 = S.launch_count()
    with Server(hbm_budget_bytes=budget, dtype=p.dtype, **kw) as srv:
        ts = [srv.submit(p, X0, V0, th, 12, snapshots=3) for _ in range(count)]
        res = [t.wait() for t in ts]
        return res, srv.stats(), S.launch_count() - n0


# states on tiles (packed: of any size), and FP64 pairs (not in the packed engine)
@pytest.mark.parametrize("packed,dtype,nx,ny,states,least", [
    (True, "f32", 30, 20, 2, 195), (False, "f32", 150, 120, 3, 195),
    (False, "f64", 30, 20, 3, 1290)])
def test_lists_are_charged_and_given_up(packed, dtype, nx, ny, states, least):
    req = request(nx, ny, dtype)
    N = nx * ny
    (full,), roomy, with_lists = serve(req, packed, 8 << 30)
    # the largest budget that leaves no room for the lists
    (lean,), tight, without = serve(req, packed, roomy["peak_bytes"] - 1)
    assert tight["completed"] == 1
    assert roomy["peak_bytes"] - tight["peak_bytes"] >= states * least * N
    for k in ("gX", "gV", "gtheta"):
        assert np.array_equal(full[k], lean[k]), k
    assert full["J"] == lean["J"]
    if dtype == "f32":  # lists from a restored state's masks are launches of their own
        assert with_lists != without


def test_admitted_bytes_include_the_lists():
    """Room for two requests but not for their lists: admitted within the budget."""
    req = request(60, 50, "f32")
    _, one, _ = serve(req, True, 8 << 30)
    _, bare, _ = serve(req, True, one["peak_bytes"] - 1)
    budget = 2 * bare["peak_bytes"] + 1
    res, st, _ = serve(req, True, budget, count=4)
    assert st["completed"] == 4 and st["peak_bytes"] <= budget
    for r in res[1:]:
        assert np.array_equal(r["gX"], res[0]["gX"])
