"""FP32 states whose particles have more neighbours than a list holds run the mask-walk
kernels, where tiles would walk the masks too and be slower: the rule on h, m, rho0 and skin,
for single states, batches and the packed server, by what a step launches."""
import ctypes as C

import numpy as np
import pytest

import cases as K

pytestmark = pytest.mark.gpu

S = pytest.importorskip("sphadjoint_gb300")
from sphadjoint_gb300 import _lib as LB  # noqa: E402


def block(nx, ny, hfac):
    dx = 0.01
    p = K.dambreak_params(dx=dx, col_h=ny * dx, Lx=2.0 * nx * dx, Ly=1.25 * max(nx, ny) * dx)
    p["h"] = hfac * dx
    rng = np.random.default_rng(nx)
    return p, K.lattice_block(nx, ny, dx, dx, dx, 0.05 * dx, rng)


def launches(step):
    """Launches of (nl_build, build_density) while step() runs."""
    L, out = S.load(), []
    LB.check(L.sph_profile_reset())
    ids = [LB.KERNEL_ID[k] for k in ("nl_build", "build_density")]
    try:
        for k in ids:
            LB.check(L.sph_profile_enable(k, 1))
        step()
        for k in ids:
            ms, n = C.c_double(), C.c_int64()
            LB.check(L.sph_profile_read(k, C.byref(ms), C.byref(n)))
            out.append(n.value)
        return tuple(out)
    finally:
        for k in ids:
            LB.check(L.sph_profile_enable(k, 0))
        LB.check(L.sph_profile_reset())


# skin 0.2: 49 neighbours are expected at h = 1.66 spacings, 50 at 1.68
@pytest.mark.parametrize("hfac,skin,tiles", [(1.3, 0.2, True), (1.66, 0.2, True),
                                             (1.68, 0.2, False), (2.5, 0.2, False),
                                             (1.3, 0.55, False)])
def test_single_states(hfac, skin, tiles):
    p, X0 = block(150, 120, hfac)
    sp = S.SPHParams(**p, dtype="f32")
    st = S.State(X0, np.zeros_like(X0), sp, skin=skin, interval=1, maxnb=128)
    th = S.DesignField(np.zeros((p["ngy"], p["ngx"])), "f32")
    assert launches(lambda: S.step(st, th)) == ((0, 1) if tiles else (1, 0))


@pytest.mark.parametrize("sizes,tiles", [((60, 20), True), ((20, 60), False)])
def test_batches_by_most_of_their_particles(sizes, tiles):
    (pa, Xa), (pb, Xb) = block(sizes[0], 30, 1.3), block(sizes[1], 30, 2.0)
    ps = [S.SPHParams(**p, dtype="f32") for p in (pa, pb)]
    bt = S.Batch([Xa, Xb], [np.zeros_like(Xa), np.zeros_like(Xb)], ps, interval=1, maxnb=128)
    th = S.BatchField([np.zeros((p["ngy"], p["ngx"])) for p in (pa, pb)], "f32")
    assert launches(lambda: S.simulate(bt, th, None, 1)) == ((0, 1) if tiles else (1, 0))


def test_server_charges_no_lists_to_such_requests():
    from sphadjoint_gb300.serve import Server

    peak = {}
    for hfac in (1.6, 1.8):
        p, X0 = block(60, 50, hfac)
        with Server(hbm_budget_bytes=4 << 30, dtype="f32", packed=True) as srv:
            srv.submit(S.SPHParams(**p, dtype="f32"), X0, np.zeros_like(X0),
                       np.zeros((p["ngy"], p["ngx"])), 4, snapshots=2, maxnb=128).wait()
            peak[hfac] = srv.stats()["peak_bytes"]
    assert peak[1.6] - peak[1.8] >= 2 * 195 * 3000
