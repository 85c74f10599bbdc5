"""The slot DTW (csrc/dtw_slots.cuh): joins whose band picks each number of
lanes per pair, cells per lane and position of the band mask, with window
lengths off the multiples of 4 and 8, against the oracle.  On the ECG-like
series most pairs reach DTW (the window table is filled), on the walk few do
(windows normalised per pair).  Tolerances of the join tests: indices exact,
distance within 1e-5 relative."""
import pytest

pytestmark = pytest.mark.gpu

# 4 lanes per pair up to w = 7, 8 up to 27, 16 up to 63 (62: a band whose last
# lane is neither empty nor walled off by its own last cell with 4 cells per
# lane of a whole warp), a whole warp above
@pytest.mark.parametrize("w", [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 13, 14, 15, 17, 19, 21, 22, 24, 25,
                               26, 27, 28, 29, 31, 33, 35, 40, 44, 47, 50, 53, 56, 58, 62, 63, 64])
def test_every_slot_layout_matches_the_oracle(gpu_dtwj, oracle, synth, w):
    with gpu_dtwj.Context() as ctx:
        for kind, n, m in (("ecg", 700, 101), ("walk", 900, 130)):
            x = (synth.ecg_like if kind == "ecg" else synth.random_walk)(n, 100 + w)
            ref = oracle.join(x, m, w)
            r = ctx.join(x, m, w)
            assert (r.i, r.j) == (ref.i, ref.j), kind
            assert abs(r.dist - ref.dist) <= max(1e-5 * ref.dist, 1e-9), kind


def test_windows_too_long_for_slots(gpu_dtwj, oracle, synth):
    # a narrow band over long windows takes more lanes per pair, in the end a
    # whole warp; the shortest windows a join takes
    for n, m, w in ((9000, 3001, 3), (5000, 1500, 10), (60, 8, 2), (60, 9, 8)):
        x = synth.random_walk(n, 7)
        ref = oracle.join(x, m, w)
        r = gpu_dtwj.join(x, m, w)
        assert (r.i, r.j) == (ref.i, ref.j), (m, w)
        assert abs(r.dist - ref.dist) <= max(1e-5 * ref.dist, 1e-9), (m, w)
