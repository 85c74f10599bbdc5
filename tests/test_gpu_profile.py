"""The matrix profile's walk (csrc/mp.cu k_profile) at sizes around its tiles
(4,032 rows, 896 lags, stages of 224 rows), with flat stretches, exact repeats
and windows without a partner, against plain FP64: distances within 1e-7 (the
direct FP64 distance against a matrix product's), indices equal wherever the
two nearest partners differ by more than that, and the lower one on exact
repeats."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reference(x, m):
    w = np.lib.stride_tricks.sliding_window_view(x, m)
    mu, sd = w.mean(1, keepdims=True), w.std(1, keepdims=True)
    flat = w.max(1) == w.min(1)  # (a constant window's computed deviation rounds)
    z = (w - mu) / np.where(flat[:, None], 1.0, sd)
    s = len(z)
    mp, mpi = np.full(s, np.inf), np.full(s, -1)
    gap = np.full(s, np.inf)
    idx = np.arange(s)
    for i in range(s):
        if flat[i]:
            continue
        c = z @ z[i]
        c[flat | (np.abs(idx - i) < m)] = -np.inf
        near = np.argsort(-c, kind="stable")[:2]
        if not np.isfinite(c[near[0]]):
            continue
        d = [np.sqrt(((z[i] - z[j]) ** 2).sum()) if np.isfinite(c[j]) else np.inf for j in near]
        k = 0 if (d[0], near[0]) <= (d[1], near[1]) else 1
        mp[i], mpi[i], gap[i] = d[k], near[k], abs(d[1] - d[0])
    return mp, mpi, gap


@pytest.mark.parametrize("n,m,kind", [(17, 8, "walk"), (130, 64, "walk"), (1000, 16, "walk"),
                                      (896 + 2 * 32, 32, "walk"), (4032 + 128, 64, "walk"),
                                      (4300, 100, "flat"), (3000, 32, "repeat"), (2500, 500, "walk")])
def test_profile_matches_fp64(gpu_dtwj, synth, n, m, kind):
    x = synth.random_walk(n, n + m)
    if kind == "flat":
        x[n // 3:n // 3 + 150] = x[n // 3]
        x[-130:] = x[-130]
    if kind == "repeat":
        x[2000:2400] = x[500:900]  # windows 500.. and 2000.. are bitwise equal
    mp, mpi = gpu_dtwj.matrix_profile(x, m)
    ref, refi, gap = _reference(x, m)
    np.testing.assert_array_equal(np.isfinite(mp), np.isfinite(ref))
    ok = np.isfinite(ref)
    np.testing.assert_allclose(mp[ok], ref[ok], rtol=1e-7, atol=1e-7)
    sure = ok & (gap > 1e-6)
    np.testing.assert_array_equal(mpi[sure], refi[sure])
    assert (mpi[~ok] == -1).all()
    if kind == "repeat":
        assert mpi[500] == 2000 and mpi[2000] == 500 and mp[500] <= 1e-7
