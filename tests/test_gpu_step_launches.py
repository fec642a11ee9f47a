"""step() runs the weights and the resampling in one launch and moves the parents' states in
the resampling block up to 1024 parents, by two grid-wide kernels above: bit for bit what
predict(), update() and resample() give, at the edges of warps, blocks and that limit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 33, 1023, 1024, 1025, 1500])
@pytest.mark.parametrize("precision", [0, 1])
def test_step_equals_its_three_calls(pkg, n, precision):
    S = pkg.scene
    sc = S.make_scene(n_landmarks=8, n_frames=5, clutter_rate=2.0, seed=S.scene_seed(0, 92))
    cfg = S.filter_config(n, 16, 32, 2.0, precision=precision, calib=sc.calib, seed=4, particles_per_feature=12)
    one, three = pkg.SCPHDCameraCalibration(cfg), pkg.SCPHDCameraCalibration(cfg)
    resampled = 0
    for z, fixed in zip(sc.frames, sc.fixed):
        u, v, d = (np.ascontiguousarray(z[:, i]) for i in range(3))
        one.step(S.DT, u, v, fixed, d)
        three.predict(S.DT)
        three.update(u, v, fixed, d)
        resampled += three.resample()
        for a, b in zip(one.particles(), three.particles()):
            np.testing.assert_array_equal(a, b)
        np.testing.assert_array_equal(one.map_sizes(), three.map_sizes())
        np.testing.assert_array_equal(one.map_weights(n - 1), three.map_weights(n - 1))
        np.testing.assert_array_equal(one.counters(), three.counters())
        c = one.counters_by_name()
        assert c["units_last_update"] <= c["units_total"] and c["survivors_last_update"] <= c["survivors_total"]
    assert n < 2 or resampled > 0
    c = one.counters_by_name()
    assert c["resamplings"] == resampled and c["frames_updated"] == 5
