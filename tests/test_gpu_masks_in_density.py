"""Small single states build the neighbour masks of a fresh cell list inside the next
step's density pass. At the sizes where the form changes (particles per block of the
FP64 pairs, the last one that does, one-launch and larger cell lists) and with rows
that spill or overflow maxnb, the state after two steps, its rows and flags equal
those of the same steps with the masks built by a launch of their own
(build_neighbors before every step), bit for bit."""
import numpy as np
import pytest

import cases as K

pytestmark = pytest.mark.gpu

S = pytest.importorskip("sphadjoint_gb300")


def _state(n, dtype, maxnb, crowd):
    rng = np.random.default_rng(n)
    p = K.dambreak_params()
    d = p["h"] / 1.3
    nx = int(np.sqrt(n))
    k = np.arange(n)
    X = np.vstack([0.02 + d * (k % nx), 0.02 + d * (k // nx)])
    X += 0.1 * d * rng.standard_normal(X.shape)
    if crowd:
        X[:, : n // 6] = X[:, :1] + 0.4 * d * rng.random((2, n // 6))
    V = 0.05 * rng.standard_normal(X.shape)
    sp = S.SPHParams(**p, dtype=dtype)
    return S.State(X, V, sp, skin=0.2, interval=1, maxnb=maxnb), sp


# FP64: 4 particles a block at 5 and 1216, 8 at 2432, 9 (not in the density pass) at
# 2433; cell lists of one launch up to 4096
@pytest.mark.parametrize("n", [5, 1216, 2432, 2433, 4100])
@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("maxnb,crowd", [(64, False), (64, True), (24, True), (100, True)])
def test_masks_built_in_the_density_pass(n, dtype, maxnb, crowd):
    a, sp = _state(n, dtype, maxnb, crowd)
    b, _ = _state(n, dtype, maxnb, crowd)
    theta = np.random.default_rng(1).random((sp.ngx, sp.ngy)) * 5.0
    for _ in range(2):
        S.step(a, theta)
        S.build_neighbors(b)
        S.step(b, theta)
    for x, y in zip(a.get(), b.get()):
        assert np.array_equal(np.asarray(x), np.asarray(y), equal_nan=True)
    assert a.take_flags() == b.take_flags()
    (ai, an), (bi, bn) = a.neighbors(), b.neighbors()
    assert np.array_equal(an, bn)
    for i in range(n):
        assert np.array_equal(ai[i, : an[i]], bi[i, : bn[i]]), i
