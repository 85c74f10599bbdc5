"""Windows whose deviation is 1e-12 of their level, the least that is not flat:
sums of the samples as they are round by a thousandth of the deviation, so the
bounds must not be built from them.  The series holds two pairs of three-level
windows on the same level in noise; the levels are chosen so that the rounding
of plain sums over 32 samples puts the closer pair's block means further apart
than the windows are.  Without seeds and with 16 tiles to a chunk the other
pair is found first.  Against the oracle: indices exact, distance within 1e-5
relative (the tolerance of the join tests)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

M, B, LEVEL, UNIT = 1024, 32, 2.0 ** 40, 2.0 ** -12
# (base, first, second) level in units, their blocks, where the two windows are
NEAR = ((-8, 5412, -5613), (-6, 24, -6), (3, 13, 13), (6000, 14000))
FAR = ((-34, -6330, 6244), (-7, 18, 2), (6, 10, 10), (2000, 4000))


def _series():
    rng = np.random.default_rng(3)
    x = rng.integers(-20 * 4096, 20 * 4096, 20000).astype(np.float64)
    for levels, step, (n0, n1, n2), at in (NEAR, FAR):
        for k, p in enumerate(at):
            base, first, second = np.array(levels) + k * np.array(step)
            x[p:p + M + 7] = base
            x[p + n0 * B:p + (n0 + n1) * B] = first
            x[p + (n0 + n1) * B:p + (n0 + n1 + n2) * B] = second
    return LEVEL + x * UNIT


def test_join_of_small_deviations_on_a_high_level(gpu_dtwj, oracle):
    x = _series()
    ref = oracle.join(x, M, 0)
    assert 6000 <= ref.i <= 6007 and ref.j - ref.i == 8000
    with gpu_dtwj.Context() as ctx:
        for chunk in (16, 0):
            ctx.set_tuning(0, chunk)
            for fl in (gpu_dtwj.F_NO_SEED, 0):
                r = ctx.join(x, M, 0, fl)
                assert (r.i, r.j) == (ref.i, ref.j), (chunk, fl)
                assert abs(r.dist - ref.dist) <= 1e-5 * ref.dist, (chunk, fl)


@pytest.mark.parametrize("level", [2.0 ** 20, 2.0 ** 30, 2.0 ** 36])
@pytest.mark.parametrize("n,m,w", [(2504, 200, 0), (3000, 64, 3), (5000, 256, 13)])
def test_join_does_not_depend_on_the_level(gpu_dtwj, oracle, synth, level, n, m, w):
    # samples on a grid of 2^-10, so that a level of up to 2^36 is added exactly
    x = np.round(synth.random_walk(n, n + m) * 1024.0) / 1024.0
    ref = oracle.join(x, m, w)
    with gpu_dtwj.Context() as ctx:
        for fl in (0, gpu_dtwj.F_MASKED_CASCADE, gpu_dtwj.F_MASKED_CASCADE | gpu_dtwj.F_NO_SEED):
            r = ctx.join(x + level, m, w, fl)
            assert (r.i, r.j) == (ref.i, ref.j), fl
            assert abs(r.dist - ref.dist) <= 1e-5 * ref.dist, fl
