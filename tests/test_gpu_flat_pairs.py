"""FP64 passes with one lane per pair (the default of FP64 states) against one
thread per particle: the same pairs, operations and summation order, so the same
bits. Sizes around a block's particles (4 to 32) and pairs (chunks of 384), spilled
rows, rows truncated at maxnb, particles the pair lists cannot hold (maxnb > 64),
particles without neighbours, batches, restored snapshots and the Tait EOS."""
import numpy as np
import pytest

import cases as K
from runners import linear_seeds, run_gpu

pytestmark = pytest.mark.gpu

S = pytest.importorskip("sphadjoint_gb300")


def block(nx, ny, hfac=1.3, outside=0, eos=0, lone=0):
    dx = 0.01
    p = K.dambreak_params(dx=dx, col_h=ny * dx, Lx=2.0 * (nx + 30) * dx,
                          Ly=1.25 * max(nx, ny, 8) * dx)
    p["h"] = hfac * dx
    if eos:
        p.update(eos=1, gamma=7)
    rng = np.random.default_rng(nx * 31 + ny)
    X0 = K.lattice_block(nx, ny, dx, dx, dx, 0.05 * dx, rng)
    X0[:, :outside] -= 0.03  # beyond the walls
    X0[0, X0.shape[1] - lone:] += 20 * dx * (1 + np.arange(lone))  # away from the rest
    V0 = 0.2 * rng.standard_normal(X0.shape)
    return dict(p=p, X0=X0, V0=V0, theta=20.0 * rng.random((p["ngy"], p["ngx"])),
                cX=rng.standard_normal(X0.shape), cV=rng.standard_normal(X0.shape))


# (case, steps, rebuild interval, maxnb, snapshots)
CASES = {
    "one": (lambda: block(1, 1), 3, 2, 64, 0),
    "five": (lambda: block(5, 1), 4, 2, 64, 0),
    "lone": (lambda: block(9, 7, lone=2), 4, 2, 64, 0),
    "240": (lambda: block(12, 20), 9, 2, 64, 0),
    "1217": (lambda: block(1217 // 31, 31, outside=4), 7, 4, 64, 0),      # 4 a block
    "5000": (lambda: block(100, 50), 6, 4, 64, 3),                          # 17 a block
    "19881": (lambda: block(141, 141), 5, 4, 64, 0),                         # 32 a block
    "spilled": (lambda: block(30, 30, hfac=3.0), 4, 2, 64, 0),
    "spilled-maxnb96": (lambda: block(30, 30, hfac=3.0), 4, 2, 96, 2),
    "long-rows-maxnb96": (lambda: block(30, 30, hfac=2.0), 4, 2, 96, 0),  # > 64 candidates
    "truncated": (lambda: block(30, 30, hfac=1.6), 4, 2, 30, 0),
    "tait": (lambda: block(40, 33, eos=1), 6, 4, 64, 0),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_flat_equals_one_thread_per_particle(name):
    make, n, interval, maxnb, snapshots = CASES[name]
    case = make()
    out = {}
    try:
        for lanes in (1, 0):
            S.set_group_lanes(lanes)
            out[lanes] = run_gpu(case, n, seeds=linear_seeds(case), interval=interval,
                                 maxnb=maxnb, snapshots=snapshots)
    finally:
        S.set_group_lanes(0)
    assert out[0]["flags"] == out[1]["flags"] and out[0]["bflags"] == out[1]["bflags"]
    assert np.all(np.isfinite(out[0]["gX"]))
    for k in ("X", "V", "gX", "gV", "gtheta"):
        assert np.array_equal(out[0][k], out[1][k]), k


def test_flat_batch_equals_solo_runs():
    """Blocks that span instances (sizes from 1 to 1600 particles)."""
    cases = [block(1, 1), block(7, 5), block(40, 40), block(3, 11), block(31, 9, eos=1)]
    ps = [S.SPHParams(**c["p"]) for c in cases]
    bt = S.Batch([c["X0"] for c in cases], [c["V0"] for c in cases], ps, interval=2)
    th = S.BatchField([c["theta"] for c in cases])
    tp = S.Tape(bt.N, 5, ps[0])
    S.simulate(bt, th, None, 5, tp)
    ws = S.BatchWorkspace(bt)
    S.batch_backward(ws, tp, th, [c["cX"] for c in cases], [c["cV"] for c in cases], interval=2)
    for c, (X, V), (gX, gV, gt) in zip(cases, bt.get(), ws.get()):
        r = run_gpu(c, 5, seeds=linear_seeds(c), interval=2)
        for a, k in ((X, "X"), (V, "V"), (gX, "gX"), (gV, "gV"), (gt, "gtheta")):
            assert np.array_equal(a, r[k]), k
