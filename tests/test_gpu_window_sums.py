"""Window sums staged through shared memory (csrc/prep.cu k_stats, k_rowterms):
windows shorter than, equal to and longer than a stage (1,024 samples), with
series that end inside a block of 256 windows, on white noise and on a series
with a flat stretch, where the diagonal bound reads them in every tile.  The
joins against the oracle: indices exact, distance within 1e-5 relative; the
mean and deviation through the matrix profile against plain FP64, 1e-7."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(2 * 8 + 3, 8), (900, 255), (2 * 1023 + 257, 1023), (2 * 1024 + 256, 1024),
         (2 * 1025 + 130, 1025), (2 * 2049 + 77, 2049)]


def _series(n, m, kind):
    x = np.random.default_rng(n).standard_normal(n)
    if kind == "flat":
        x[n // 4:n // 4 + m + 5] = 1e3
    return x


@pytest.mark.parametrize("n,m", SIZES)
@pytest.mark.parametrize("kind", ["noise", "flat"])
def test_join_matches_oracle(gpu_dtwj, oracle, n, m, kind):
    x, w = _series(n, m, kind), max(1, m // 50)
    ref = oracle.join(x, m, w)
    with gpu_dtwj.Context() as ctx:
        for fl in (0, gpu_dtwj.F_MASKED_CASCADE):
            r = ctx.join(x, m, w, fl)
            assert (r.i, r.j) == (ref.i, ref.j), fl
            assert abs(r.dist - ref.dist) <= max(1e-5 * ref.dist, 1e-9), fl


@pytest.mark.parametrize("n,m", SIZES)
def test_profile_matches_fp64(gpu_dtwj, n, m):
    x = _series(n, m, "noise")
    mp, _ = gpu_dtwj.matrix_profile(x, m)
    w = np.lib.stride_tricks.sliding_window_view(x, m)
    z = (w - w.mean(1, keepdims=True)) / w.std(1, keepdims=True)
    for i in range(0, len(z), 41):
        j = np.r_[0:max(0, i - m + 1), i + m:len(z)]
        if not len(j):
            assert np.isinf(mp[i])
            continue
        ref = np.sqrt(((z[j] - z[i]) ** 2).sum(1).min())
        assert abs(mp[i] - ref) <= 1e-7 * (1 + ref), i
