"""Small single states, and FP32 states on tiles, build the neighbour masks of a fresh
cell list inside the next step's density pass. At the sizes where the form changes (particles per block of the
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
        c = min(n // 6, 1000)
        X[:, :c] = X[:, :1] + 0.4 * d * rng.random((2, c))
    V = 0.05 * rng.standard_normal(X.shape)
    sp = S.SPHParams(**p, dtype=dtype)
    return S.State(X, V, sp, skin=0.2, interval=1, maxnb=maxnb), sp


def _same(a, b):
    for x, y in zip(a.get(), b.get()):
        assert np.array_equal(np.asarray(x), np.asarray(y), equal_nan=True)
    assert a.take_flags() == b.take_flags()
    (ai, an), (bi, bn) = a.neighbors(), b.neighbors()
    assert np.array_equal(an, bn)
    for i in range(an.size):
        assert np.array_equal(ai[i, : an[i]], bi[i, : bn[i]]), i


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
    _same(a, b)


# tiles of 128: a whole number of them and one particle more; rows above a list's 48
# entries and windows above their 640 slots (crowded) fall back to the masks
@pytest.mark.parametrize("n", [16512, 16513])
@pytest.mark.parametrize("maxnb,crowd", [(64, False), (24, False), (64, True), (100, True)])
def test_masks_and_lists_built_in_the_density_pass_of_tiles(n, maxnb, crowd):
    a, sp = _state(n, "f32", maxnb, crowd)
    b, _ = _state(n, "f32", maxnb, crowd)
    theta = np.random.default_rng(1).random((sp.ngx, sp.ngy)) * 5.0
    for _ in range(2):
        S.step(a, theta)
        S.build_neighbors(b)
        S.step(b, theta)
    _same(a, b)
