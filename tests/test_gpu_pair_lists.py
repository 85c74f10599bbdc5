"""Pair lists (dtwj_pair_dtw, dtwj_pair_dtw_noalloc) over the layouts their rule
picks: FP64 by window length and band, FP32 by the length of the list (one pair
per warp up to 2,368 pairs), against the oracle.  Tolerances of the pair-DTW
parity tests: FP64 1e-10, FP32 2e-4 relative."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,w", [(8, 0), (9, 8), (33, 2), (64, 4), (128, 7), (200, 20), (256, 13),
                                 (512, 52), (300, 103), (520, 255), (3000, 30), (7000, 3)])
def test_pair_lists_match_the_oracle(gpu_dtwj, oracle, synth, m, w):
    import torch

    n = max(2 * m + 1, m + 1200)
    x = synth.random_walk(n, m)
    rng = np.random.default_rng(w)
    base = rng.integers(0, n - m + 1, (2, 12))
    ref = np.array([oracle.pair_dist(x, m, w, int(i), int(j)) for i, j in base.T])
    lib = gpu_dtwj.load()
    xd = torch.from_numpy(x).cuda()
    for count in (12, 2368, 2369):
        pi, pj = (np.resize(b, count).astype(np.int64) for b in base)
        for precise, rtol in ((True, 1e-10), (False, 2e-4)):
            d = gpu_dtwj.pair_dtw(x, m, w, pi, pj, precise=precise)
            np.testing.assert_allclose(d, np.resize(ref, count), rtol=rtol, atol=1e-9)
            pid, pjd = torch.from_numpy(pi).cuda(), torch.from_numpy(pj).cuda()
            out = torch.empty(count, dtype=torch.float64, device="cuda")
            vp = ctypes.c_void_p
            rc = lib.dtwj_pair_dtw_noalloc(vp(xd.data_ptr()), n, m, w, vp(pid.data_ptr()),
                                           vp(pjd.data_ptr()), count, int(precise),
                                           vp(out.data_ptr()), None)
            assert rc == gpu_dtwj.OK
            torch.cuda.synchronize()
            np.testing.assert_allclose(out.cpu().numpy(), np.resize(ref, count), rtol=rtol, atol=1e-9)
