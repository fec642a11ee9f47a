"""Components of the merge's "may merge" graph of every size class, against the oracle's greedy
merge: up to 8 members (one thread), a warp's edges, hundreds, and all of the largest list in
one component; survivors of a component lie scattered over the list.

Means are whole numbers and covariances the identity, so squared distances are multiples of a
half and min_separation = 6.25 is never met: membership is exact in both precisions.  Merged
values are sums of up to `size` members of at most 64 in size: size * 64 * 2^-24 in FP32,
size * 64 * 2^-52 in FP64, times 4 for the divisions and the covariance's difference.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(8, 1, 9), (31, 32, 33, 7), (64, 65, 2, 160), (161, 9, 9, 9), (700, 300, 40, 5), (2048,)],
                         ids=str)
@pytest.mark.parametrize("precision", [0, 1])
def test_components_of_all_sizes_match_the_oracle(pkg, orc, sizes, precision):
    rng = np.random.default_rng(sum(sizes))
    n = sum(sizes)
    comps = np.zeros((n, 28))
    comps[:, 0] = rng.integers(1, 64, n) / 64.0   # ties among them
    comps[:, 1:4] = rng.integers(0, 7, (n, 3))
    comps[:, 4:7] = rng.integers(0, 3, (n, 3))
    comps[:, 1] += np.repeat(np.arange(len(sizes)) * 100, sizes)
    comps[:, 7 + np.array([0, 2, 5, 9, 14, 20])] = 1.0
    comps = comps[rng.permutation(n)]
    flags = (rng.uniform(size=n) < 0.02).astype(np.uint8)
    ref, ref_member = orc.merge(comps, flags, 6.25)
    out, member = pkg.merge_components(comps, flags, 6.25, precision)
    assert np.array_equal(member, ref_member)
    assert out.shape == ref.shape
    eps = 2.0 ** (-24 if precision == pkg.SCPHD_FP32 else -52)
    # a component's u offset of up to 300 carries its own rounding
    np.testing.assert_allclose(out, ref, rtol=16 * eps, atol=4 * max(sizes) * 64 * eps)
