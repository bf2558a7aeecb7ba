"""Iterative density weights over the transposed tap matrix: against their FP64
restatement, with samples in two bins (the later bin's weight stays), an empty
bin and samples at the faces of the grid."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("img,grid,nch", [((16, 16, 12), (32, 32, 24), 1), ((24, 20, 16), (40, 32, 24), 4),
                                          ((64, 16, 12), (128, 32, 24), 4)])
def test_density_weights_match_restatement(gpu_lib, cgs, oracle_mod, o64, img, grid, nch):
    rng = np.random.default_rng(3)
    k = rng.uniform(0.0, 1.0, (900, 3))
    k[:4] = [[0, 0, 0], [1, 1, 1], [0, 1, 0], [1, 0, 1]]
    bins = [np.arange(0, 500), np.zeros(0, np.int64), np.arange(400, 900)]   # 400..499 in two bins
    p = oracle_mod.make_params(img, grid, nch, kb_w=4.0, kb_b=9.0)
    taps = o64.taps(p, k)
    want = oracle_mod.pipe_menon(taps, int(np.prod(grid)), 5, bins)
    r = cgs.Reco(img, grid, nch, kb_w=4.0, kb_b=9.0)
    r.set_trajectory(k)
    r.set_bins(bins)
    got = r.pipe_menon_dcf(5)
    # 5 iterations of FP32 sums of at most a few hundred terms: 1e-5 (the
    # restatement's own weights are float)
    assert rel_l2(got, want) < 1e-5
    assert np.array_equal(got, r.pipe_menon_dcf(5))
