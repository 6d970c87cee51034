"""FP32 pair passes over neighbour lists and staged windows against the mask
walks (the "mask" density form runs every pass as a mask walk). Both visit the
same pairs in the same order with the same operations, so results are the same
bits: tiles of one and of several cell rows, partial last tiles, rows beyond the
64-slot masks and particles with more candidates than a list holds (which take
the mask walk inside a tile), tiles whose window does not fit, restored
snapshots (lists made from the masks), batches, and the model variants."""
import numpy as np
import pytest

import cases as K
from runners import linear_seeds, run_gpu

pytestmark = pytest.mark.gpu

S = pytest.importorskip("sphadjoint_gb300")


def seeded(case, seed=3):
    rng = np.random.default_rng(seed)
    case["cX"] = rng.standard_normal(case["X0"].shape)
    case["cV"] = rng.standard_normal(case["X0"].shape)
    return case


def block(nx, ny, hfac=1.3, jitter=0.05, outside=0):
    dx = 0.01
    p = K.dambreak_params(dx=dx, col_h=ny * dx, Lx=2.0 * nx * dx, Ly=1.25 * max(nx, ny) * dx)
    p["h"] = hfac * dx
    rng = np.random.default_rng(nx * 31 + ny)
    X0 = K.lattice_block(nx, ny, dx, dx, dx, jitter * dx, rng)
    X0[:, :outside] -= 0.03  # beyond the walls
    V0 = 0.2 * rng.standard_normal(X0.shape)
    return seeded(dict(p=p, X0=X0, V0=V0, theta=20.0 * rng.random((p["ngy"], p["ngx"]))))


def tait(case):
    case["p"] = dict(case["p"], eos=1, gamma=7, visc=1, alpha=0.02)
    return case


# (case, steps, rebuild interval, maxnb, snapshots)
CASES = {
    "one-row-tiles": (lambda: block(150, 9), 6, 4, 64, 0),
    "many-row-tiles": (lambda: block(7, 90), 6, 2, 64, 0),        # runs of ~22 particles
    "too-many-runs": (lambda: block(2, 300), 5, 2, 64, 0),        # no window: mask walk
    "partial-tile": (lambda: block(43, 3, outside=5), 6, 3, 64, 0),
    "one-particle": (lambda: block(1, 1), 3, 2, 64, 0),
    "long-lists": (lambda: block(40, 40, hfac=1.75), 5, 2, 96, 0),  # ~55 candidates
    "spilled-rows": (lambda: block(30, 30, hfac=3.0), 4, 2, 64, 0),
    "truncated-lists": (lambda: block(40, 40, hfac=1.5), 5, 2, 30, 0),
    "restored": (lambda: block(60, 50), 17, 4, 64, 3),
    "tait-av": (lambda: tait(block(60, 50)), 8, 4, 64, 0),
    "tait-av-restored": (lambda: tait(block(61, 33)), 11, 4, 64, 2),
}


@pytest.fixture
def forms():
    S.set_group_lanes(1)
    yield S.set_density_form
    S.set_density_form("pairs")
    S.set_group_lanes(0)


@pytest.mark.parametrize("name", sorted(CASES))
def test_lists_equal_the_mask_walks(forms, name):
    make, n, interval, maxnb, snapshots = CASES[name]
    case = make()
    out = {}
    for f in ("mask", "pairs"):
        forms(f)
        out[f] = run_gpu(case, n, dtype="f32", seeds=linear_seeds(case), interval=interval,
                         maxnb=maxnb, snapshots=snapshots)
    assert out["mask"]["flags"] == out["pairs"]["flags"]
    assert np.all(np.isfinite(out["pairs"]["gX"]))
    for k in ("X", "V", "gX", "gV", "gtheta"):
        assert np.array_equal(out["pairs"][k], out["mask"][k]), k


def test_batch_lists_equal_the_mask_walks(forms):
    """Tiles that span several instances (sizes from 1 to 2000 particles)."""
    cases = [block(1, 1), block(7, 5), block(50, 40), block(3, 11), block(31, 9)]
    ps = [S.SPHParams(**c["p"], dtype="f32") for c in cases]
    out = {}
    for f in ("mask", "pairs"):
        forms(f)
        bt = S.Batch([c["X0"] for c in cases], [c["V0"] for c in cases], ps, interval=2)
        th = S.BatchField([c["theta"] for c in cases], "f32")
        tp = S.Tape(bt.N, 6, ps[0])
        S.simulate(bt, th, None, 6, tp)
        ws = S.BatchWorkspace(bt)
        S.batch_backward(ws, tp, th, [c["cX"] for c in cases], [c["cV"] for c in cases],
                         interval=2)
        out[f] = [a for m in bt.get() + ws.get() for a in m]
    for a, b in zip(out["mask"], out["pairs"]):
        assert np.array_equal(a, b)
