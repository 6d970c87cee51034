"""Steps on a stream that the caller is recording with the CUDA API go into the caller's
graph kernel by kernel. A state's first step there allocates nothing (the lists of its pair
passes are taken at a later step that runs): the graph can be replayed again and again, and
steps outside it follow, all with the bits of the same steps made directly."""
import ctypes as C

import numpy as np
import pytest

import cases as K

pytestmark = pytest.mark.gpu

S = pytest.importorskip("sphadjoint_gb300")
torch = pytest.importorskip("torch")


@pytest.fixture
def stream():
    from sphadjoint_gb300 import _lib as LB
    s = torch.cuda.Stream()
    LB.check(S.load().sph_set_stream(C.c_void_p(s.cuda_stream)))
    yield s
    torch.cuda.synchronize()
    LB.check(S.load().sph_set_stream(None))


def case(nx, ny, dtype):
    dx = 0.01
    p = K.dambreak_params(dx=dx, col_h=ny * dx, Lx=2.0 * nx * dx, Ly=1.25 * max(nx, ny) * dx)
    rng = np.random.default_rng(nx + ny)
    X0 = K.lattice_block(nx, ny, dx, dx, dx, 0.05 * dx, rng)
    sp = S.SPHParams(**p, dtype=dtype)
    return (lambda: S.State(X0, 0.2 * np.ones_like(X0), sp, interval=2),
            S.DesignField(20.0 * rng.random((p["ngy"], p["ngx"])), dtype))


# tiles, lane groups in FP32; pairs with and without the masks in the density pass
@pytest.mark.parametrize("dtype,nx,ny", [("f32", 150, 120), ("f32", 40, 30), ("f64", 40, 30),
                                         ("f64", 90, 60)])
def test_first_steps_inside_a_callers_recording(stream, dtype, nx, ny):
    new, th = case(nx, ny, dtype)
    st, ref = new(), new()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        for _ in range(4):  # two rebuilds and four steps: the state's buffers end as they began
            S.step(st, th)
    for replay in range(3):
        graph.replay()
        torch.cuda.synchronize()
        for _ in range(4):
            S.step(ref, th)
        for a, b in zip(st.get(), ref.get()):
            assert np.array_equal(a, b), replay
    for _ in range(5):  # outside the graph
        S.step(st, th)
        S.step(ref, th)
    for a, b in zip(st.get(), ref.get()):
        assert np.array_equal(a, b)
