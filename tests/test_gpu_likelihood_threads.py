"""The likelihood with one and with two measurements a thread (many FP32 parents), and blocks that
spill over: more than 1024 measurements for the stage kernels, more than 256 for the fused one.

Normalisers of the first parents have to be bit for bit those of a filter of few parents, which
takes one measurement a thread (parents of equal index draw the same streams), and of its fused
update's, where that fits the same FP32 rows.

Against 64-bit values: quadratic forms of terms that count are at most 40; their FP32 error is
that of S^-1 by cofactors, 16 eps times the condition of S scaled to unit diagonal, which is
asserted to be at most 10: 40 * 16 * 6e-8 * 10 / 2 = 2e-4; log and sum add parts in 10^6.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _filter(pkg, n, cap, precision, seed=9):
    S = pkg.scene
    sc = S.make_scene(n_landmarks=40, n_frames=2, clutter_rate=8.0, seed=S.scene_seed(0, 96))
    cfg = S.filter_config(n, 24, cap, 8.0, precision=precision, calib=sc.calib, seed=seed, particles_per_feature=16)
    cfg.max_survivors = 3 * 24 + cap
    return sc, cfg, pkg.SCPHDCameraCalibration(cfg)


def _more(rng, cfg, z, m):
    extra = rng.random((max(0, m - len(z)), 3)) * [2 * cfg.u0, 2 * cfg.v0, 40.0] + [0.0, 0.0, 5.0]
    return np.ascontiguousarray(np.concatenate([z, extra])[:m])


@pytest.mark.parametrize("m", [1, 32, 33, 64, 65, 128, 161, 1024, 1030, 1090])
@pytest.mark.parametrize("precision", [0, 1])
def test_many_parents_equal_few(pkg, precision, m):
    rng = np.random.default_rng(m)
    sc, cfg, _ = _filter(pkg, 12, 1120, precision)
    out = []
    for n, fused in ((12, 0), (4000, 0), (12, 1)):
        if fused and precision == 0 and m > 32:
            continue   # the FP32 fused build may contract differently: compared below
        _, _, f = _filter(pkg, n, 1120, precision)
        f.set_fused(fused)
        for z in (sc.frames[0], sc.frames[1]):
            z = _more(np.random.default_rng(m), cfg, z, m)
            f.predict(pkg.scene.DT)
            f.update(z[:, 0], z[:, 1], True, z[:, 2])
        ell, ll = f.normalizers(m)
        out.append([ell[:12], ll[:12], f.map_sizes()[:12]] + [f.mixture(pkg.SCPHD_MIX_MERGED, p) for p in range(12)])
        f.close()
    for other in out[1:]:
        for a, b in zip(out[0], other):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("fused", [0, 1])
@pytest.mark.parametrize("m", [257, 600])
def test_fused_blocks_spill_over(pkg, fused, m):
    """FP32, fused and staged: 64-bit normalisers from the rows the update fitted."""
    _check_exact(pkg, 12, m, fused)


@pytest.mark.parametrize("n,m", [(12, 30), (4000, 64), (4000, 160), (12, 1030)])
def test_normalisers_in_64_bits(pkg, n, m):
    _check_exact(pkg, n, m, 0)


def _check_exact(pkg, n, m, fused):
    rng = np.random.default_rng(n + m)
    sc, cfg, f = _filter(pkg, n, 1120, pkg.SCPHD_FP32)
    f.set_fused(fused)
    G, P = 24, 16
    depth = rng.uniform(3.0, 8.0, n * G)
    centre = np.stack([rng.uniform(-0.3, 0.3, n * G) * depth, rng.uniform(-0.2, 0.2, n * G) * depth, depth,
                       *rng.normal(0, 0.02, (3, n * G))], axis=1)
    spread = np.array([0.01, 0.01, 0.02, 0.02, 0.02, 0.02])
    state = (np.tile(sc.calib, (n, 1)), np.full(n, -np.log(n)), np.full(n, G, np.int32), rng.uniform(0.3, 1.0, n * G),
             centre[:, :, None] + spread[:, None] * rng.standard_normal((n * G, 6, P)), np.full((n * G, P), 1.0 / P))
    f.set_state(*state)
    f.update(np.zeros(1), np.zeros(1), False, np.zeros(1))
    fits = [f.mixture(pkg.SCPHD_MIX_FITTED, p) for p in range(12)]
    noise = np.diag([cfg.std_u ** 2, cfg.std_v ** 2, cfg.std_d ** 2])
    # measurements about the first parents' Gaussians, so that their terms count
    at = np.concatenate([x[:, 2:5] for x in fits])
    z = at[rng.integers(len(at), size=m)] + rng.standard_normal((m, 3)) * 2.0 * np.sqrt(np.diag(noise))
    z = np.ascontiguousarray(np.abs(z))
    f.set_state(*state)
    f.update(z[:, 0], z[:, 1], False, z[:, 2])
    ell, _ = f.normalizers(m)
    counted = 0
    for p in range(12):
        fit = f.mixture(pkg.SCPHD_MIX_FITTED, p)
        lw = np.empty((len(fit), m))
        for j, row in enumerate(fit):
            cov = np.zeros((6, 6))
            cov[np.tril_indices(6)] = row[8:]
            s = cov[:3, :3] + np.tril(cov[:3, :3], -1).T + noise
            d = np.sqrt(np.diag(s))
            assert np.linalg.cond(s / np.outer(d, d)) <= 10
            nu = z - row[2:5]
            lw[j] = (np.log(row[0] * row[1]) - 1.5 * np.log(2 * np.pi) - 0.5 * np.linalg.slogdet(s)[1]
                     - 0.5 * np.einsum("mi,ij,mj->m", nu, np.linalg.inv(s), nu))
        rest = np.log(m * cfg.w0 + cfg.kappa)
        ref = np.logaddexp(np.logaddexp.reduce(lw, 0), rest)
        counted += int((ref > rest + 1.0).sum())
        np.testing.assert_allclose(ell[p], ref, rtol=0, atol=2e-4)
    assert counted > m // 2   # a measurement lies near one parent's Gaussians: most of them decide a normaliser
    f.close()
