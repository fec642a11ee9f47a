"""The packed single-precision cloud fit (the stage kernels') and the one-sample-per-lane form (the
fused update's) have to give the same bits: fitted rows and clouds, at the edges of the packed
layout, with carried and drawn clouds, samples of zero weight and a pending prediction; and the
packed normals the same as the one-sample ones, finite for every uniform."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", [1, 3, 4, 5, 31, 32, 33, 50, 63, 64, 65, 97, 100, 127, 128, 129, 200, 255, 256])
@pytest.mark.parametrize("zeros", [False, True])
def test_both_forms_fit_the_same_rows(pkg, P, zeros):
    S = pkg.scene
    n, G = 4, 70
    sc = S.make_scene(n_landmarks=30, n_frames=3, clutter_rate=6.0, seed=S.scene_seed(0, 90))
    cfg = S.filter_config(n, G, 96, 6.0, precision=pkg.SCPHD_FP32, calib=sc.calib, seed=3, particles_per_feature=P)
    cfg.pd = 1.0 if zeros else 0.95
    rng = np.random.default_rng(P)
    depth = rng.uniform(3.0, 8.0, n * G)
    centre = np.stack([rng.uniform(-0.6, 0.6, n * G) * depth, rng.uniform(-0.45, 0.45, n * G) * depth, depth,
                       *rng.normal(0, 0.02, (3, n * G))], axis=1)
    spread = np.array([0.03, 0.03, 0.06, 0.02, 0.02, 0.02])
    om = np.full((n * G, P), 1.0 / P)
    if zeros:
        om[::3] = 0.0
        om[1::3, ::2] = 0.0
    state = (np.tile(sc.calib, (n, 1)) + rng.normal(0, 0.02, (n, 12)), np.full(n, -np.log(n)), np.full(n, G, np.int32),
             rng.uniform(0.05, 1.0, n * G), centre[:, :, None] + spread[:, None] * rng.standard_normal((n * G, 6, P)), om)
    fs = []
    for fused in (0, 1):
        f = pkg.SCPHDCameraCalibration(cfg)
        f.set_fused(fused)
        f.set_state(*state)
        fs.append(f)
    for k in range(2):   # carried clouds, then drawn ones among them
        z = sc.frames[k]
        for f in fs:
            if k or not zeros:
                f.predict(S.DT)
            f.update(z[:, 0], z[:, 1], False, z[:, 2])
        for p in range(n):
            a, b = (f.mixture(pkg.SCPHD_MIX_FITTED, p) for f in fs)
            np.testing.assert_array_equal(a, b)
        for x, y in zip(*(f.map_clouds(0) for f in fs)):
            np.testing.assert_array_equal(x, y)


def test_packed_normals(tmp_path):
    lib = str(tmp_path / "libnormals.so")
    nvcc = os.environ.get("NVCC") or "/usr/local/cuda/bin/nvcc"
    csrc = os.path.join(ROOT, "scphd-camera-calibration_b200", "csrc")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                    "-I", csrc, "-I", os.path.join(ROOT, "include"), "-o", lib,
                    os.path.join(ROOT, "tests", "cpp", "normals_check.cu")], check=True)
    bad = (ctypes.c_ulonglong * 2)()
    assert ctypes.CDLL(lib).check_normals(bad) == 0
    assert list(bad) == [0, 0]
