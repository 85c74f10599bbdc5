"""Seeds of joins of 1,024 tiles and more, which the group bound finds
(csrc/group.cu) unless it settles too little: the best seed must be the one a
walk over every diagonal finds.  A small chunk leaves no room for the group
bound's lists, so the same join then walks.  The two choose among the same
pairs by keys of 20 bits and agree on the closest, whose DTW is the same FP32
arithmetic: equal up to its rounding (1e-6 relative).  White noise, on which
the bound settles nothing, must not pay for it: a sample finds that out in a
small part of a walk's time, and three walks' time is allowed (the lists took
eight)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _series(synth, kind, n, seed):
    if kind == "walk":
        return synth.random_walk(n, seed)
    rng = np.random.default_rng(seed)
    if kind == "noise":
        return rng.standard_normal(n)
    if kind == "motif":
        x = rng.standard_normal(n)
        x[n // 3:n // 3 + 300] = synth.random_walk(300, seed)
        x[n - 20000:n - 19700] = x[n // 3:n // 3 + 300] + 0.01 * rng.standard_normal(300)
        return x
    x = np.convolve(rng.standard_normal(n + 64), np.hanning(65), "valid")[:n]  # "smooth"
    return x


# both group sizes (8 from m = 512 on); random walks also at a window so short that
# the bound leaves too much
@pytest.mark.parametrize("kind,n,m,w", [
    ("walk", 100003, 256, 13), ("walk", 95001, 1024, 20), ("walk", 100003, 64, 3),
    ("smooth", 100003, 256, 13), ("smooth", 95001, 512, 10), ("noise", 100003, 64, 0),
    ("noise", 95001, 512, 0), ("motif", 100003, 256, 0)])
def test_group_seeds_are_those_of_a_walk(gpu_dtwj, synth, kind, n, m, w):
    x = _series(synth, kind, n, n + m)
    k = gpu_dtwj.PHASES.index("profile")
    with gpu_dtwj.Context() as ctx:
        runs = [ctx.join(x, m, w, gpu_dtwj.F_PROFILE) for _ in range(4)]
        ctx.set_tuning(0, 64)
        walks = [ctx.join(x, m, w, gpu_dtwj.F_PROFILE) for _ in range(4)]
    r, p = runs[0], walks[0]
    assert np.isfinite(r.seed_bsf)
    assert abs(r.seed_bsf - p.seed_bsf) <= 1e-6 * p.seed_bsf
    assert (r.i, r.j) == (p.i, p.j) and abs(r.dist - p.dist) <= 1e-9
    if kind in ("noise", "motif"):
        assert min(q.phase_seconds[k] for q in runs) <= 3 * min(q.phase_seconds[k] for q in walks)


def test_join_of_noise_without_the_group_bound(gpu_dtwj, oracle):
    # 128 tiles and more: the sweep samples the bound too, and leaves every tile dense
    x = np.random.default_rng(9).standard_normal(45000)
    ref = oracle.join(x, 128, 0)
    with gpu_dtwj.Context() as ctx:
        for fl in (0, gpu_dtwj.F_NO_SEED, gpu_dtwj.F_MASKED_CASCADE):
            r = ctx.join(x, 128, 0, fl)
            assert (r.i, r.j) == (ref.i, ref.j), fl
            assert abs(r.dist - ref.dist) <= 1e-5 * ref.dist, fl
            total = (r.pruned_fast + r.pruned_paa + r.pruned_kim + r.pruned_masked +
                     r.pruned_keogh + r.dtw_calls)
            assert 0 <= total - r.pairs <= 700, (fl, total, r.pairs)
