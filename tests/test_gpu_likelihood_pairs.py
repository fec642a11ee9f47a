"""The likelihood takes two Gaussians at a time in FP32: normalisers and survivors against their
64-bit values from the same fitted rows, at odd and even map sizes (an odd one's last pair is
half empty), at the edges of a warp of measurements, and with more candidates per measurement
than the list holds (wide noise: nearly every pair survives).

Tolerance of a normaliser, FP32: terms within 20 of the largest count, their quadratic forms are
at most 40 and carry the rounding of S^-1 (cofactors: a few eps times a condition number of up
to 1e3), 1e-3 * 40 / 2 = 2e-2 at most; FP64: 1e-9.  Survivors whose weight is within five times
that of min_weight (wide noise: quadratic forms of up to 140) may fall on either side.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G,M,wide", [(1, 1, False), (2, 31, False), (3, 33, False), (16, 20, True), (17, 20, True),
                                      (33, 20, True), (64, 32, False), (65, 150, False), (127, 64, False)])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("precision", [0, 1])
def test_normalisers_and_survivors(pkg, G, M, wide, dim, precision):
    n, P = 5, 16
    sc = pkg.scene.make_scene(n_landmarks=30, n_frames=1, clutter_rate=6.0, seed=pkg.scene.scene_seed(0, 94))
    cfg = pkg.scene.filter_config(n, 128, 160, 6.0, precision=precision, calib=sc.calib, seed=5,
                                  particles_per_feature=P, meas_dim=dim)
    cfg.std_u = cfg.std_v = 60.0 if wide else 6.0
    cfg.std_d = 20.0 if wide else 3.0
    cfg.min_weight = 1e-30 if wide else 1e-3
    cfg.max_survivors = 1200
    rng = np.random.default_rng(100 * G + M)
    f = pkg.SCPHDCameraCalibration(cfg)
    depth = rng.uniform(3.0, 8.0, n * G)
    centre = np.stack([rng.uniform(-0.3, 0.3, n * G) * depth, rng.uniform(-0.2, 0.2, n * G) * depth, depth,
                       *rng.normal(0, 0.02, (3, n * G))], axis=1)
    spread = np.array([0.03, 0.03, 0.06, 0.02, 0.02, 0.02])
    clouds = centre[:, :, None] + spread[:, None] * rng.standard_normal((n * G, 6, P))
    sizes = np.full(n, G, np.int32)
    sizes[1] = max(1, G - 1)   # the other parity beside it
    keep = np.concatenate([np.arange(p * G, p * G + sizes[p]) for p in range(n)])
    f.set_state(np.tile(sc.calib, (n, 1)), np.full(n, -np.log(n)), sizes, rng.uniform(0.05, 1.0, n * G)[keep],
                clouds[keep], np.full((len(keep), P), 1.0 / P))
    z = rng.random((M, 3)) * [2 * cfg.u0, 2 * cfg.v0, 40.0] + [0.0, 0.0, 5.0]
    f.update(np.ascontiguousarray(z[:, 0]), np.ascontiguousarray(z[:, 1]), False,
             np.ascontiguousarray(z[:, 2]) if dim == 3 else None)
    ell, _ = f.normalizers(M)
    tol = 2e-2 if precision == pkg.SCPHD_FP32 else 1e-9
    noise = np.diag([cfg.std_u ** 2, cfg.std_v ** 2, cfg.std_d ** 2][:dim])
    least = most = 0
    for p in range(n):
        fit = f.mixture(pkg.SCPHD_MIX_FITTED, p)
        assert len(fit) == sizes[p]
        lw = np.full((len(fit), M), -np.inf)
        for j, row in enumerate(fit):
            cov = np.zeros((6, 6))
            cov[np.tril_indices(6)] = row[8:]
            s = cov[:dim, :dim] + np.tril(cov[:dim, :dim], -1).T + noise
            if row[0] * row[1] > 0:
                nu = z[:, :dim] - row[2:2 + dim]
                lw[j] = (np.log(row[0] * row[1]) - 0.5 * dim * np.log(2 * np.pi) - 0.5 * np.linalg.slogdet(s)[1]
                         - 0.5 * np.einsum("mi,ij,mj->m", nu, np.linalg.inv(s), nu))
        ref = np.log(np.exp(lw).sum(0) + M * cfg.w0 + cfg.kappa)
        np.testing.assert_allclose(ell[p], ref, rtol=0, atol=tol)
        w = np.concatenate([lw - ref, (np.log(cfg.w0) - ref)[None]]) - np.log(cfg.min_weight)
        least += (w > 5 * tol).sum()
        most += (w > -5 * tol).sum()
    assert least <= f.counters_by_name()["survivors_last_update"] <= most
    assert not wide or most > n * M * G * 0.8
