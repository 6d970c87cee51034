"""The lane and density settings are process-wide, and results do not depend on the ones
chosen here (FP64: any lane setting; FP32 states with one thread per particle: mask walks or
tiles). So a solve gives the same bits while another thread moves the setting all the time:
each step reads it once, and its launches agree on who builds the masks of a fresh cell
list and who loads the next tape state."""
import itertools
import threading

import numpy as np
import pytest

import cases as K
from runners import linear_seeds, run_gpu

pytestmark = pytest.mark.gpu

S = pytest.importorskip("sphadjoint_gb300")


def block(nx, ny):
    dx = 0.01
    p = K.dambreak_params(dx=dx, col_h=ny * dx, Lx=2.0 * nx * dx, Ly=1.25 * max(nx, ny) * dx)
    rng = np.random.default_rng(nx * 31 + ny)
    X0 = K.lattice_block(nx, ny, dx, dx, dx, 0.05 * dx, rng)
    return dict(p=p, X0=X0, V0=0.2 * rng.standard_normal(X0.shape),
                theta=20.0 * rng.random((p["ngy"], p["ngx"])),
                cX=rng.standard_normal(X0.shape), cV=rng.standard_normal(X0.shape))


class Moving:
    """Moves a setting through its values from a second thread."""

    def __init__(self, move, values):
        self.move, self.values, self.stop, self.moves = move, values, False, 0

    def __enter__(self):
        self.thread = threading.Thread(target=self.run)
        self.thread.start()
        return self

    def run(self):
        for v in itertools.cycle(self.values):
            if self.stop:
                break
            self.move(v)
            self.moves += 1

    def __exit__(self, *exc):
        self.stop = True
        self.thread.join()


@pytest.fixture(autouse=True)
def defaults():
    yield
    S.set_group_lanes(0)
    S.set_density_form("pairs")


# FP64: masks built by the density pass (up to 2432 particles) and before it
@pytest.mark.parametrize("dtype,nx,ny", [("f64", 30, 25), ("f64", 70, 40), ("f32", 150, 120)])
@pytest.mark.parametrize("interval,snapshots", [(1, 0), (2, 0), (2, 4)])
def test_a_moving_setting_leaves_the_results(dtype, nx, ny, interval, snapshots):
    case = block(nx, ny)
    args = dict(dtype=dtype, seeds=linear_seeds(case), interval=interval, snapshots=snapshots)
    want = run_gpu(case, 40, **args)
    move, values = ((S.set_group_lanes, (0, 1, 16, 32)) if dtype == "f64"
                    else (S.set_density_form, ("pairs", "mask")))
    with Moving(move, values) as m:
        for _ in range(6):
            got = run_gpu(case, 40, **args)
            assert got["flags"] == want["flags"] and got["bflags"] == want["bflags"]
            for k in ("X", "V", "gX", "gV", "gtheta"):
                assert np.array_equal(got[k], want[k]), k
    assert m.moves > 100


def test_a_moving_setting_leaves_the_results_of_a_batch():
    cases = [block(60, 40), block(7, 5), block(31, 29)]
    ps = [S.SPHParams(**c["p"], dtype="f32") for c in cases]

    def solve():
        bt = S.Batch([c["X0"] for c in cases], [c["V0"] for c in cases], ps, interval=1)
        th = S.BatchField([c["theta"] for c in cases], "f32")
        tp = S.Tape(bt.N, 30, ps[0])
        S.simulate(bt, th, None, 30, tp)
        ws = S.BatchWorkspace(bt)
        S.batch_backward(ws, tp, th, [c["cX"] for c in cases], [c["cV"] for c in cases], interval=1)
        return [a for m in bt.get() + ws.get() for a in m]

    want = solve()
    with Moving(S.set_density_form, ("pairs", "mask")):
        for _ in range(6):
            for a, b in zip(want, solve()):
                assert np.array_equal(a, b)
