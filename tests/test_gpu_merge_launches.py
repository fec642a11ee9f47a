"""A filter whose survivor capacity leaves an SM one merge block merges its parents in two
launches, one sized for the usual parent and one for those with more survivors.  A filter of
few parents takes one launch; parents 0..n-1 of both draw the same streams, so with a fixed
camera (no resampling) their maps have to be equal bit for bit.

Wide measurement noise makes nearly every (Gaussian, measurement) pair survive: parents cross
the first launch's capacity (about 1000) while their maps fill, so both launches, the counting
order (at most 160 survivors) and the sorts are used."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_two_merge_launches_equal_one(pkg, precision):
    S = pkg.scene
    sc = S.make_scene(n_landmarks=60, n_frames=6, clutter_rate=20.0, seed=S.scene_seed(0, 91))
    sizes = []
    runs = {}
    for n in (400, 12):
        cfg = S.filter_config(n, 24, 96, 20.0, precision=precision, calib=sc.calib, seed=9, particles_per_feature=32)
        cfg.std_u = cfg.std_v = 60.0
        cfg.std_d = 20.0
        cfg.min_weight = 1e-9
        cfg.max_survivors = 1600
        f = pkg.SCPHDCameraCalibration(cfg)
        out = []
        for k in range(6):
            z = sc.frames[2 * (k // 2)]
            m = (5, 20, 35, 45, 50, 55)[k]   # from a few survivors to most of the capacity
            f.predict(S.DT)
            f.update(z[:m, 0], z[:m, 1], True, z[:m, 2])
            out += [f.mixture(which, p) for which in (pkg.SCPHD_MIX_FITTED, pkg.SCPHD_MIX_MERGED) for p in range(12)]
            out += [f.map_weights(p) for p in range(12)] + [f.normalizers(m)[1][:12]]
            if n == 400:
                sizes.append(f.counters_by_name()["survivors_last_update"] / n)
        c = f.counters_by_name()
        assert c["scratch_overflows"] == 0
        runs[n] = out
    assert min(sizes) < 160 and max(sizes) > 1050, sizes
    for a, b in zip(runs[400], runs[12]):
        np.testing.assert_array_equal(a, b)
