"""Results of every size class -- within the parents' page-locked rows, up to the filter's largest
result, past what is page-locked -- one after another from one filter, against the asynchronous
copies, an independent sum and a filter that is asked in the other order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,G,P", [(1, 4, 1), (1, 12, 8), (40, 96, 100), (40, 128, 200), (700, 12, 8)])
@pytest.mark.parametrize("precision", [0, 1])
def test_results_of_all_sizes(pkg, n, G, P, precision):
    S = pkg.scene
    sc = S.make_scene(n_landmarks=20, n_frames=4, clutter_rate=2.0, seed=S.scene_seed(0, 95))
    cfg = S.filter_config(n, G, 96, 2.0, precision=precision, calib=sc.calib, seed=8, particles_per_feature=P)
    fs = [pkg.SCPHDCameraCalibration(cfg) for _ in range(2)]
    for z, fixed in zip(sc.frames, sc.fixed):
        for f in fs:
            f.predict(S.DT)
            f.update(z[:, 0], z[:, 1], fixed, z[:, 2])
    m = len(sc.frames[-1])
    asks = [lambda f: f.particles(), lambda f: (f.map_sizes(),), lambda f: (f.counters(),), lambda f: f.normalizers(m),
            lambda f: f.map_clouds(n - 1), lambda f: (f.map_weights(n - 1),), lambda f: f.particles()]
    a = [ask(fs[0]) for ask in asks]
    b = [ask(fs[1]) for ask in reversed(asks)][::-1]
    for x, y in zip(a, b):
        for u, v in zip(x, y):
            np.testing.assert_array_equal(u, v)
    ell, ll = a[3]
    for p in (0, n - 1):
        w = fs[0].mixture(pkg.SCPHD_MIX_FITTED, p)[:, 0].sum()
        assert abs(ell[p].sum() + w - ll[p]) <= 1e-9 * max(1.0, abs(ll[p]))
    x, om = a[4]
    assert x.shape == (len(om), 6, P) and len(om) == a[1][0][n - 1] == len(a[5][0])
    assert np.isfinite(x).all() and ((om >= 0) & (om <= 1)).all()
