"""The objectives of a batch go out in groups of 32 instances: J and the seeds (read
back as the gradient of one step) of every instance equal those it gives alone, bit
for bit, for batches of two, a full group, a group and one, and more than two, with
instances of one particle and around a block's 256."""
import numpy as np
import pytest

import cases as K

pytestmark = pytest.mark.gpu

S = pytest.importorskip("sphadjoint_gb300")

SIZES = [1, 255, 256, 257, 600]


@pytest.mark.parametrize("count", [2, 32, 33, 70])
@pytest.mark.parametrize("kind", ["ke_right", "target"])
def test_objective_of_a_group(count, kind):
    p = K.dambreak_params()
    sp = S.SPHParams(**p)
    rng = np.random.default_rng(count)
    d = p["h"] / 1.3
    X0, V0, th, args = [], [], [], []
    for b in range(count):
        n = SIZES[b % len(SIZES)]
        k = np.arange(n)
        X0.append(np.vstack([0.6 * p["Lx"] + d * (k % 25), 0.02 + d * (k // 25)]) - 0.01 * b)
        V0.append(rng.standard_normal((2, n)))
        th.append(5.0 * rng.random((sp.ngx, sp.ngy)))
        args.append([0.5 + 0.01 * b, 0.1, 0.2])
    use = args if kind == "target" else None
    bt = S.Batch(X0, V0, [sp] * count, interval=2)
    field = S.BatchField(th)
    tape = S.Tape(bt.N, 1, sp)
    S.simulate(bt, field, None, 1, tape)
    ws = S.BatchWorkspace(bt)
    J = ws.objective(bt, kind, use)
    S.batch_backward(ws, tape, field, interval=2, seeded=True)
    grads = ws.get()
    for b in range(count):
        st = S.State(X0[b], V0[b], sp, interval=2)
        t1 = S.Tape(st.N, 1, sp)
        S.simulate(st, th[b], None, 1, t1)
        w1 = S.AdjointWorkspace(st.N, sp)
        assert J[b] == w1.objective(st, kind, args[b] if use else None)
        S.backward_seeded(w1, t1, th[b], sp, interval=2)
        for x, y in zip(grads[b], w1.get()):
            assert np.array_equal(x, y)
