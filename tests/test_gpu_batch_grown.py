"""A batch stepped until its maps have grown: past the steps on which it times its launch shapes
(every merge width and cloud-fit split), the capture of its graph and replays with changing
measurement counts, one frame empty.  Every member has to end where it gets alone, bit for bit.

One member's parents have more survivors than a merge launch sized for the usual parent holds
(wide noise: nearly every pair survives), so that the launch for the listed ones runs as well."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _frame(z, m, dim, fixed):
    z = z[:m]
    return z[:, 0], z[:, 1], z[:, 2] if dim == 3 else None, fixed


def members(pkg, precision, dim, wide):
    """(scene, configuration, measurements of a frame or None for all of them)"""
    S = pkg.scene
    out = []
    for i, (n, g, m) in enumerate([(130, 96, 96), (7, 64, 64)]):
        sc = S.make_scene(n_landmarks=14 + 6 * i, n_frames=16, clutter_rate=4.0, seed=S.scene_seed(5, 20 + i))
        cfg = S.filter_config(n, g, m, 4.0, precision=precision, calib=sc.calib, seed=40 + i,
                              particles_per_feature=40 + 60 * i, meas_dim=dim)
        out.append((sc, cfg, None))
    sc = S.make_scene(n_landmarks=60, n_frames=6, clutter_rate=20.0, seed=S.scene_seed(0, 91))
    cfg = S.filter_config(wide, 24, 96, 20.0, precision=precision, calib=sc.calib, seed=9, particles_per_feature=32,
                          meas_dim=dim)
    cfg.std_u = cfg.std_v = 60.0
    cfg.std_d = 20.0
    cfg.min_weight = 1e-9
    cfg.max_survivors = 1600
    out.append((sc, cfg, (5, 20, 35, 45, 50, 55)))
    return out


def frames(ms, k, dim):
    out = []
    for i, (sc, cfg, counts) in enumerate(ms):
        j = k % (2 * sc.n_frames - 2)
        j = j if j < sc.n_frames else 2 * sc.n_frames - 2 - j
        z = sc.frames[j]
        m = counts[k % len(counts)] if counts else (0 if i == 1 and k == 25 else len(z))
        out.append(_frame(z, m, dim, sc.fixed[j]))
    return out


def assert_same(alone, batched, what):
    for i, (a, b) in enumerate(zip(alone, batched)):
        for x, y, name in zip(a.particles(), b.particles(), ("states", "log-weights")):
            assert np.array_equal(x, y), f"{what} member {i}: {name}"
        assert np.array_equal(a.map_sizes(), b.map_sizes()), f"{what} member {i}: map sizes"
        assert np.array_equal(a.resample_indices(), b.resample_indices()), f"{what} member {i}: resampling"
        for p in range(0, a.n_parents, 13):
            assert np.array_equal(a.mixture(1, p), b.mixture(1, p)), f"{what} member {i}: merged, parent {p}"
            assert np.array_equal(a.map_weights(p), b.map_weights(p)), f"{what} member {i}: map, parent {p}"


@pytest.mark.parametrize("use_graph", [False, True])
@pytest.mark.parametrize("precision,dim", [(0, 3), (1, 3), (1, 2)])
def test_grown_batch_equals_its_members_alone(pkg, precision, dim, use_graph):
    ms = members(pkg, precision, dim, 400)
    alone = [pkg.SCPHDCameraCalibration(c) for _, c, _ in ms]
    batched = [pkg.SCPHDCameraCalibration(c) for _, c, _ in ms]
    for f in alone:
        f.set_autotune(False)
    batch = pkg.SCPHDBatch(batched, use_graph=use_graph)
    launches, most = [], 0.0
    for k in range(32):
        fr = frames(ms, k, dim)
        for f, (u, v, d, fixed) in zip(alone, fr):
            f.step(pkg.scene.DT, u, v, fixed_camera=fixed, d=d)
        before = pkg.kernel_launches()
        batch.step(pkg.scene.DT, fr)
        launches.append(pkg.kernel_launches() - before)
        most = max(most, alone[2].counters_by_name()["survivors_last_update"] / 400)
        if k < 2 or k >= 15:
            assert_same(alone, batched, f"frame {k}")
    assert batch.fit_split()["fit_tuned"]
    assert most > 1050 and max(launches) == 7, (most, launches)   # parents were listed, and merged by the second launch
    batch.close()
    for f in alone + batched:
        assert f.counters_by_name()["scratch_overflows"] == 0
        f.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_resident_batch_takes_one_merge_launch(pkg, precision):
    """Parents that are all resident at the full survivor capacity are merged in one launch."""
    ms = members(pkg, precision, 3, 12)[1:]
    alone = [pkg.SCPHDCameraCalibration(c) for _, c, _ in ms]
    batched = [pkg.SCPHDCameraCalibration(c) for _, c, _ in ms]
    batch = pkg.SCPHDBatch(batched)
    for k in range(8):
        fr = frames(ms, k, 3)
        for f, (u, v, d, fixed) in zip(alone, fr):
            f.step(pkg.scene.DT, u, v, fixed_camera=fixed, d=d)
        before = pkg.kernel_launches()
        batch.step(pkg.scene.DT, fr)
        assert pkg.kernel_launches() - before == 6
    assert_same(alone, batched, "last")
    batch.close()


def _step_all(pkg, ms, alone, batch, k):
    fr = frames(ms, k, 3)
    for f, (u, v, d, fixed) in zip(alone, fr):
        f.step(pkg.scene.DT, u, v, fixed_camera=fixed, d=d)
    batch.step(pkg.scene.DT, fr)


@pytest.mark.parametrize("precision", [0, 1])
def test_rebuilt_batch_goes_on_with_its_members_shapes(pkg, precision):
    """Batches made anew from the same filters, as a server makes them: trials are carried on, a
    choice is kept, and a young member neither holds back nor spoils the others."""
    ms = members(pkg, precision, 3, 30)
    alone = [pkg.SCPHDCameraCalibration(c) for _, c, _ in ms]
    batched = [pkg.SCPHDCameraCalibration(c) for _, c, _ in ms]
    batch = pkg.SCPHDBatch(batched[:2], use_graph=True)
    for k in range(18):   # 16 frames, two of the six trials
        _step_all(pkg, ms[:2], alone[:2], batch, k)
    assert not batch.fit_split()["fit_tuned"]
    batch.set_fit_split(2)   # open until the shapes are settled: the graph of the first steps goes
    _step_all(pkg, ms[:2], alone[:2], batch, 18)
    batch.close()
    batch = pkg.SCPHDBatch(batched, use_graph=True)   # with a young third member of fewer parents
    tuned = []
    for k in range(19, 26):
        _step_all(pkg, ms, alone, batch, k)
        tuned.append(batch.fit_split()["fit_tuned"])
    assert tuned == [False] * 4 + [True] * 3   # four more trials, seen on the step after them
    split = batch.fit_split()
    batch.close()
    batch = pkg.SCPHDBatch(batched, use_graph=True)
    assert batch.fit_split() == split
    for k in range(26, 31):
        _step_all(pkg, ms, alone, batch, k)
    assert_same(alone, batched, "rebuilt")
    batch.close()


def test_settled_batch_refuses_other_shapes(pkg):
    ms = members(pkg, 0, 3, 30)[:2]
    alone = [pkg.SCPHDCameraCalibration(c) for _, c, _ in ms]
    batched = [pkg.SCPHDCameraCalibration(c) for _, c, _ in ms]
    batch = pkg.SCPHDBatch(batched, use_graph=True)
    for k in range(24):
        _step_all(pkg, ms, alone, batch, k)
    with pytest.raises(pkg.ScphdError):
        batch.set_fit_split(4)
    with pytest.raises(pkg.ScphdError):
        batch.set_fused(1)
    batch.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_served_long_jobs_equal_jobs_alone(pkg, precision):
    """Jobs that outlive the tuning, with others arriving and retiring beside them."""
    S = pkg.scene
    jobs = []
    for i, (n, nf) in enumerate([(96, 40), (64, 33), (40, 9), (30, 12), (50, 27)]):
        sc = S.make_scene(n_landmarks=12 + 2 * i, n_frames=nf, clutter_rate=4.0, seed=S.scene_seed(4, 30 + i))
        jobs.append((sc, S.filter_config(n, 96, 64, 4.0, precision=precision, calib=sc.calib, seed=800 + i,
                                         particles_per_feature=36 + 8 * i)))
    srv = pkg.SCPHDServer(int(2e9), precision=precision, meas_dim=3, use_graph=True)
    arrive = {0: [0, 1], 5: [2], 19: [3], 25: [4]}
    ids = {}
    for it in range(60):
        for i in arrive.get(it, []):
            ids[i] = srv.submit(jobs[i][1], jobs[i][0].frames, jobs[i][0].fixed, S.DT)
        srv.step()
    srv.drain()
    assert srv.stats()["done"] == len(jobs) and srv.stats()["rebuilds"] >= 5
    for i, (sc, cfg) in enumerate(jobs):
        f = pkg.SCPHDCameraCalibration(cfg)
        for k, z in enumerate(sc.frames):
            f.step(S.DT, z[:, 0], z[:, 1], fixed_camera=sc.fixed[k], d=z[:, 2])
        for x, y in zip(srv.result(ids[i]), f.particles()):
            assert np.array_equal(x, y), f"job {i}"
    srv.close()
