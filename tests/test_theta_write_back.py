"""The theta write-back summed per design cell in a warp: the integer pieces it
adds (host check of the shipped header), and dJ/dtheta on design grids from one
cell for all particles to several cells per particle (more than the eight
cells a warp sums, where each lane adds its own)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import cases as K

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "sphadjoint_gb300", "csrc")


def test_parts_and_limbs_equal_the_fixed_point_integers(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("g++ not found")
    exe = str(tmp_path / "fixed_parts_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", CSRC,
                    os.path.join(HERE, "fixed_parts_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("nt", [2, 7, 40, 300])
@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_gradient_on_coarse_and_fine_design_grids(dtype, nt):
    """The node sums are exact integers, so they do not depend on which lanes
    share a warp: FP64 with one thread per particle (warp sums) equals one group
    per particle (per-particle adds) bit for bit; in FP32, where the two forms
    round galpha differently, a solo run equals the same instance in a batch
    behind 13 other particles, whose warps hold other lanes."""
    from runners import linear_seeds, run_gpu
    import sphadjoint_gb300 as S

    case = K.adjoint_case(seed=nt)
    rng = np.random.default_rng(nt)
    case["p"] = dict(case["p"], ngx=nt, ngy=max(2, nt - 1))
    case["theta"] = 3 * rng.random((max(2, nt - 1), nt))
    seeds = linear_seeds(case)
    try:
        S.set_group_lanes(1)
        one = run_gpu(case, 8, dtype=dtype, seeds=seeds)
        if dtype == "f64":
            S.set_group_lanes(16)
            other = run_gpu(case, 8, dtype=dtype, seeds=seeds)["gtheta"]
        else:
            few = K.adjoint_case(seed=1)
            few = {k: few[k][:, :13] if k in ("X0", "V0", "cX", "cV") else few[k] for k in few}
            two = [few, case]
            ps = [S.SPHParams(**c["p"], dtype=dtype) for c in two]
            bt = S.Batch([c["X0"] for c in two], [c["V0"] for c in two], ps, interval=1)
            th = S.BatchField([c["theta"] for c in two], dtype)
            tp = S.Tape(bt.N, 8, ps[0])
            S.simulate(bt, th, None, 8, tp)
            ws = S.BatchWorkspace(bt)
            S.batch_backward(ws, tp, th, [c["cX"] for c in two], [c["cV"] for c in two],
                             interval=1)
            other = np.asarray(ws.get()[1][2], np.float64)
    finally:
        S.set_group_lanes(0)
    assert np.max(np.abs(one["gtheta"])) > 0
    assert np.array_equal(one["gtheta"], other)
