"""The single-precision cloud fit against a plain FP64 refit of the clouds it fits.

The map's Euclidean clouds (scphd_get_map_clouds: drawn components regenerated by another
kernel, carried clouds as stored) are projected into the parent's camera and refitted with
numpy; the next update's fitted mixture has to agree.  Sample counts cover the edges of the
kernel's layout: units of four samples, passes of 32 units, Gaussians that straddle passes,
rounds of one to sixteen Gaussians and more Gaussians per warp than a sorted batch of 32.

Tolerances, from the FP32 rounding of one projection (a few eps times coordinates of up to
1e3, against standard deviations of 0.1 and more) and of sums over at most 256 samples about
the first one (256 eps times a few squared deviations): means within 2e-3 standard
deviations, covariances within 5e-3 of sqrt(S_aa S_bb).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COUNTS = [1, 3, 4, 5, 31, 32, 33, 63, 64, 65, 97, 100, 127, 128, 129, 200, 255, 256]


def _filter(pkg, n, G, P, pd=0.95, seed=3):
    sc = pkg.scene.make_scene(n_landmarks=30, n_frames=3, clutter_rate=6.0, seed=pkg.scene.scene_seed(0, 90))
    cfg = pkg.scene.filter_config(n, G, 96, 6.0, precision=pkg.SCPHD_FP32, calib=sc.calib, seed=seed,
                                  particles_per_feature=P)
    cfg.pd = pd
    return sc, cfg, pkg.SCPHDCameraCalibration(cfg)


def _clouds(rng, n_entries, P):
    depth = rng.uniform(3.0, 8.0, n_entries)
    centre = np.stack([rng.uniform(-0.6, 0.6, n_entries) * depth, rng.uniform(-0.45, 0.45, n_entries) * depth, depth,
                       *rng.normal(0, 0.02, (3, n_entries))], axis=1)
    spread = np.array([0.03, 0.03, 0.06, 0.02, 0.02, 0.02])
    return centre[:, :, None] + spread[:, None] * rng.standard_normal((n_entries, 6, P))


def _project(pkg, x, ext, cfg):
    """(g, 6, P) world samples -> (g, 6, P) (u, v, d, vu, vv, vd)."""
    R = pkg.scene.rotation_terms(ext[6:9])
    pos = np.einsum("ij,gjp->gip", R, x[:, :3] - ext[:3, None])
    vel = np.einsum("ij,gjp->gip", R, x[:, 3:])
    iz = 1.0 / pos[:, 2]
    return np.stack([cfg.u0 - cfg.fx * pos[:, 0] * iz, cfg.v0 - cfg.fy * pos[:, 1] * iz, -cfg.fx * cfg.baseline * iz,
                     -cfg.fx * (vel[:, 0] * pos[:, 2] - vel[:, 2] * pos[:, 0]) * iz * iz,
                     -cfg.fy * (vel[:, 1] * pos[:, 2] - vel[:, 2] * pos[:, 1]) * iz * iz,
                     cfg.fx * cfg.baseline * vel[:, 2] * iz * iz], axis=1)


def _check(pkg, f, cfg, sc, frame, parents):
    """Refit the clouds f holds, update f, compare its fitted rows; returns the rows compared
    of (weighted, unweighted, out of view) fits."""
    st, _ = f.particles()
    held = {p: (f.map_clouds(p), f.map_weights(p)) for p in parents}
    z = sc.frames[frame]
    f.update(z[:, 0], z[:, 1], False, z[:, 2])
    seen = [0, 0, 0]
    P = int(cfg.particles_per_feature)
    for p in parents:
        (x, om), w = held[p]
        fit = f.mixture(pkg.SCPHD_MIX_FITTED, p)
        assert len(fit) == len(w)
        np.testing.assert_allclose(fit[:, 0], w, rtol=1e-6)
        y = _project(pkg, x, st[p], cfg)
        lim = np.array([2 * cfg.u0, 2 * cfg.v0])[None, :, None]
        inside = ((y[:, :2] >= 0) & (y[:, :2] <= lim)).all(1) & (y[:, 2] >= 0)
        edge = (np.minimum(np.abs(y[:, :2]), np.abs(y[:, :2] - lim)).min(1) < 0.01).any(1)
        for j in np.flatnonzero(~edge):
            n_in = int(inside[j].sum())
            assert fit[j, 1] == np.float32(n_in * cfg.pd / P)
            wt = om[j] * cfg.pd * inside[j]
            cov = np.zeros((6, 6))
            cov[np.tril_indices(6)] = fit[j, 8:]
            cov = cov + np.tril(cov, -1).T
            if wt.sum() > 0:
                v = wt / wt.sum()
                mean = (v * y[j]).sum(1)
                d = y[j] - mean[:, None]
                # the weights' squares are FP32 values (0 where they underflow)
                squares = np.square(wt.astype(np.float32)).astype(np.float64).sum()
                ref = (v * d) @ d.T * (1 + squares / wt.sum() ** 2)
                sd = np.sqrt(np.diag(ref)) + 1e-2 * (n_in == 1)
                assert (np.abs(fit[j, 2:8] - mean) <= 2e-3 * sd + 1e-3 * (n_in < 3)).all(), (p, j)
                assert (np.abs(cov - ref) <= 5e-3 * np.outer(sd, sd) + 1e-3 * (n_in < 3)).all(), (p, j)
                seen[0] += 1
            elif n_in > 0:   # every sample weighted 1: the sum, and the scatter about it
                total = y[j].sum(1)
                d = y[j] - total[:, None]
                ref = d @ d.T * (P * P + P) / P
                sd = np.sqrt(np.diag(ref))
                assert (np.abs(fit[j, 2:8] - total) <= 1e-4 * np.abs(y[j]).sum(1)).all(), (p, j)
                assert (np.abs(cov - ref) <= 5e-3 * np.outer(sd, sd)).all(), (p, j)
                seen[1] += 1
            else:
                assert (fit[j, 8:] == 0).all()
                seen[2] += 1
    return seen


@pytest.mark.parametrize("P", COUNTS)
@pytest.mark.parametrize("G,split", [(5, 1), (70, 1), (150, 1), (150, 4)])
def test_fit_matches_a_refit_of_the_clouds(pkg, P, G, split):
    n = 4
    sc, cfg, f = _filter(pkg, n, G, P)
    f.set_fit_split(split)
    rng = np.random.default_rng(P)
    f.set_state(np.tile(sc.calib, (n, 1)) + rng.normal(0, 0.02, (n, 12)), np.full(n, -np.log(n)),
                np.full(n, G, np.int32), rng.uniform(0.05, 1.0, n * G), _clouds(rng, n * G, P),
                np.full((n * G, P), 1.0 / P))
    first = _check(pkg, f, cfg, sc, 0, (0, n - 1))    # carried clouds only
    second = _check(pkg, f, cfg, sc, 1, (0, n - 1))   # drawn components and carried clouds
    assert first[0] > 0 and second[0] > 0


@pytest.mark.parametrize("P", [5, 64, 100, 256])
def test_fit_with_zero_and_subnormal_sample_weights(pkg, P):
    """pD = 1 and sample weights of 0: a Gaussian with none left takes the unweighted fit."""
    n, G = 3, 9
    sc, cfg, f = _filter(pkg, n, G, P, pd=1.0)
    rng = np.random.default_rng(100 + P)
    om = np.full((n * G, P), 1.0 / P)
    om[::3] = 0.0            # all zero: unweighted
    om[1::3, ::2] = 0.0      # every second one zero
    om[2::6] *= 1e-30
    f.set_state(np.tile(sc.calib, (n, 1)), np.full(n, -np.log(n)), np.full(n, G, np.int32),
                rng.uniform(0.05, 1.0, n * G), _clouds(rng, n * G, P), om)
    seen = _check(pkg, f, cfg, sc, 0, range(n))
    assert seen[0] > 0 and seen[1] > 0
    assert f.counters_by_name()["unit_weight_fits"] >= seen[1]
