"""A filter of many parents times its merge at 256, 128 and 64 threads on grown maps: every width
has to leave it where a filter with tuning off is, bit for bit.  (64 threads are tried from 889
FP32 and 593 FP64 parents on, on the updates after the twenty-second.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,n", [(0, 900), (1, 600)])
def test_merge_widths_on_grown_maps(pkg, precision, n):
    S = pkg.scene
    sc = S.make_scene(n_landmarks=40, n_frames=17, clutter_rate=10.0, seed=S.scene_seed(6, 40))
    cfg = S.filter_config(n, 64, 96, 10.0, precision=precision, calib=sc.calib, seed=63, particles_per_feature=20)
    tuned, plain = pkg.SCPHDCameraCalibration(cfg), pkg.SCPHDCameraCalibration(cfg)
    plain.set_autotune(False)
    for k in range(32):
        z = sc.frames[k if k < 17 else 32 - k]
        for f in (tuned, plain):
            f.step(S.DT, z[:, 0], z[:, 1], fixed_camera=sc.fixed[k if k < 17 else 32 - k], d=z[:, 2])
        if k < 21:
            continue
        for a, b in zip(tuned.particles(), plain.particles()):
            assert np.array_equal(a, b), f"frame {k}"
        assert np.array_equal(tuned.map_sizes(), plain.map_sizes()), f"frame {k}"
        for p in range(0, n, 37):
            assert np.array_equal(tuned.mixture(1, p), plain.mixture(1, p)), f"frame {k} parent {p}"
    s = tuned.launch_shapes()
    assert s["fit_tuned"] and s["merge_threads"] in (64, 128, 256)
    assert plain.launch_shapes()["merge_threads"] == 256
