"""FP32 tiles: particles whose cell rows exceed the 64-slot masks but whose neighbours fit a
list (what a column that presses through a wall leaves in the border cells: everything beyond
a wall is clamped into them) take lists like the others, with the bits of the mask walks, also
in tiles whose window is too large to be staged (lists of slots, up to a span of 16 bits):
from a fresh cell list, from restored snapshots, with rows cut at maxnb, in batches, with the
model variants and in the packed server."""
import numpy as np
import pytest

import cases as K
from runners import linear_seeds, run_gpu

pytestmark = pytest.mark.gpu

S = pytest.importorskip("sphadjoint_gb300")

SKIN = 0.2


def beyond(nx, ny, inside, model=None, crowd=0):
    """A block of which `inside` columns are in the tank and the rest beyond its right wall;
    the first `crowd` particles are within half a spacing's distance of each other."""
    dx = 0.01
    p = K.dambreak_params(dx=dx, col_h=ny * dx, Lx=(inside + 0.5) * dx, Ly=1.25 * ny * dx)
    p.update(kw=0.5, **(model or {}))
    rng = np.random.default_rng(nx * 31 + ny)
    X0 = K.lattice_block(nx, ny, dx, dx, dx, 0.05 * dx, rng)
    X0[:, :crowd] = X0[:, :1] + 0.5 * dx * rng.random((2, crowd))
    return dict(p=p, X0=X0, V0=0.05 * rng.standard_normal(X0.shape),
                theta=20.0 * rng.random((p["ngy"], p["ngx"])),
                cX=rng.standard_normal(X0.shape), cV=rng.standard_normal(X0.shape))


def spilled(case):
    """Particles with a row of more than 64 slots, and the largest number of neighbours."""
    p, X = case["p"], case["X0"]
    cs = 2.0 * p["h"] * (1 + SKIN)
    n = [int(np.ceil(p[k] / cs)) + 2 for k in ("Lx", "Ly")]
    cx, cy = (np.clip(np.floor(X[k] / cs).astype(int) + 2, 1, n[k]) for k in (0, 1))
    count = np.zeros((n[1] + 2, n[0] + 2), int)
    np.add.at(count, (cy, cx), 1)
    row = count[:, :-2] + count[:, 1:-1] + count[:, 2:]
    worst = np.max([row[cy + d, cx - 1] for d in (-1, 0, 1)], axis=0)
    d2 = ((X[:, :, None] - X[:, None, :]) ** 2).sum(0)
    return int((worst > 64).sum()), int((d2 < cs * cs).sum(1).max()) - 1


# (case, steps, rebuild interval, maxnb, snapshots)
TAIT_AV = dict(eos=1, gamma=7, visc=1, alpha=0.02)
CASES = {
    "fresh": (lambda: beyond(60, 30, 25), 7, 3, 64, 0),
    "every-step": (lambda: beyond(50, 31, 10), 5, 1, 64, 0),
    "restored": (lambda: beyond(60, 30, 25), 15, 4, 64, 3),
    "cut-at-maxnb": (lambda: beyond(60, 30, 25), 6, 2, 20, 0),
    "restored-cut-at-maxnb": (lambda: beyond(60, 30, 25), 15, 4, 20, 3),
    "wide": (lambda: beyond(200, 18, 4), 5, 2, 64, 0),           # no tile has a window
    "wide-restored": (lambda: beyond(120, 24, 4), 15, 4, 64, 3),
    "too-long-for-a-list": (lambda: beyond(60, 30, 25, crowd=60), 4, 2, 90, 0),
    "tait-av": (lambda: beyond(60, 30, 25, TAIT_AV), 6, 3, 64, 0),
    "tait-av-restored": (lambda: beyond(61, 30, 25, TAIT_AV), 15, 4, 64, 3),
}


@pytest.fixture
def forms():
    S.set_group_lanes(1)
    yield S.set_density_form
    S.set_density_form("pairs")
    S.set_group_lanes(0)


@pytest.mark.parametrize("name", sorted(CASES))
def test_lists_of_spilled_rows_equal_the_mask_walks(forms, name):
    make, n, interval, maxnb, snapshots = CASES[name]
    case = make()
    rows, most = spilled(case)
    assert rows > 300 and (most <= 48) == (name != "too-long-for-a-list")
    out = {}
    for f in ("mask", "pairs"):
        forms(f)
        out[f] = run_gpu(case, n, dtype="f32", seeds=linear_seeds(case), interval=interval,
                         maxnb=maxnb, snapshots=snapshots)
    assert out["mask"]["flags"] == out["pairs"]["flags"]
    assert np.all(np.isfinite(out["pairs"]["gX"]))
    for k in ("X", "V", "gX", "gV", "gtheta"):
        assert np.array_equal(out["pairs"][k], out["mask"][k]), k


def test_rows_that_span_more_than_16_bits(forms):
    """Three rows of 22,200 slots: neither a window nor 16-bit slots."""
    case = beyond(7400, 9, 3)
    out = {}
    for f in ("mask", "pairs"):
        forms(f)
        out[f] = run_gpu(case, 2, dtype="f32", seeds=linear_seeds(case), interval=2)
    for k in ("X", "V", "gX", "gV", "gtheta"):
        assert np.array_equal(out["pairs"][k], out["mask"][k]), k


@pytest.mark.parametrize("models", [({}, {}, {}), ({}, TAIT_AV, {})])
def test_lists_of_spilled_rows_in_a_batch_and_in_the_packed_server(forms, models):
    from sphadjoint_gb300.serve import Server

    cases = [beyond(*a, m) for a, m in zip([(60, 30, 25), (20, 20, 18), (70, 25, 12)], models)]
    ps = [S.SPHParams(**c["p"], dtype="f32") for c in cases]
    got = {}
    for f in ("mask", "pairs"):
        forms(f)
        bt = S.Batch([c["X0"] for c in cases], [c["V0"] for c in cases], ps, interval=3)
        th = S.BatchField([c["theta"] for c in cases], "f32")
        tp = S.Tape(bt.N, 7, ps[0])
        S.simulate(bt, th, None, 7, tp)
        ws = S.BatchWorkspace(bt)
        S.batch_backward(ws, tp, th, [c["cX"] for c in cases], [c["cV"] for c in cases], interval=3)
        got[f] = [a for m in bt.get() + ws.get() for a in m]
        with Server(hbm_budget_bytes=4 << 30, dtype="f32", packed=True) as srv:
            ts = [srv.submit(p, c["X0"], c["V0"], c["theta"], 12, snapshots=3)
                  for p, c in zip(ps, cases)]
            for r in [t.wait() for t in ts]:
                got[f] += [r["gX"], r["gV"], r["gtheta"]]
    for a, b in zip(got["mask"], got["pairs"]):
        assert np.array_equal(a, b)
