"""Results up to 512 KB come back through the filter's page-locked buffer, larger ones straight
into the caller's array: the same values on both sides of the limit, and beside a NULL array."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [100, 5041, 5042, 6000])   # 104 bytes a parent: 524264, 524368 of 524288
def test_readback_on_both_sides_of_the_staging_limit(pkg, n):
    import torch
    S = pkg.scene
    sc = S.make_scene(n_landmarks=6, n_frames=2, clutter_rate=2.0, seed=S.scene_seed(0, 93))
    cfg = S.filter_config(n, 12, 32, 2.0, precision=pkg.SCPHD_FP32, calib=sc.calib, seed=8, particles_per_feature=8)
    f = pkg.SCPHDCameraCalibration(cfg)
    for z, fixed in zip(sc.frames, sc.fixed):
        f.predict(S.DT)
        f.update(z[:, 0], z[:, 1], fixed, z[:, 2])
    m = len(sc.frames[-1])
    st, lw = f.particles()
    pst, plw = torch.zeros(n, 12, dtype=torch.float64, pin_memory=True), torch.zeros(n, dtype=torch.float64, pin_memory=True)
    f.particles_async(pst.data_ptr(), plw.data_ptr())
    f.synchronize()
    np.testing.assert_array_equal(st, pst.numpy())
    np.testing.assert_array_equal(lw, plw.numpy())
    only = np.zeros(n)   # NULL states
    lib = pkg.load_library()
    assert lib.scphd_get_particles(f._h, None, only.ctypes.data_as(ctypes.POINTER(ctypes.c_double))) == 0
    np.testing.assert_array_equal(only, lw)
    ell, ll = f.normalizers(m)
    assert ell.shape == (n, m) and np.isfinite(ell).all()
    # the parents' log-likelihoods are the normalisers' sums and the fitted weights'
    for p in (0, n // 2, n - 1):
        w = f.mixture(pkg.SCPHD_MIX_FITTED, p)[:, 0].sum()
        assert abs(ell[p].sum() + w - ll[p]) <= 1e-9 * max(1.0, abs(ll[p]))
    if not sc.fixed[-1]:
        np.testing.assert_array_equal(f.map_sizes() <= 12, True)
