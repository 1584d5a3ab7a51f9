"""Norms of a step follow the templates that the bank holds when the filter object is made: rows that a caller put there
(longer than the generator's, shorter, all zero, ending in a NaN), read from the templates themselves."""
import numpy as np
import pytest
import torch

from oracle import synth

pytestmark = pytest.mark.gpu

TLEN = 1 << 16
FLEN = TLEN // 2 + 1
DF = 2048.0 / TLEN


@pytest.mark.parametrize('flen', [1, 33, 1025, 4096, 4097, 9000])
def test_row_ends(flen):
    from gwb200 import fp_filter
    H = torch.zeros((9, flen + 3), dtype=torch.complex64, device='cuda')[:, :flen]
    want = [0, 1, flen, flen // 2 + 1, max(1, flen - 1), min(flen, 1024), max(1, flen - 4096), flen, flen]
    for i, e in enumerate(want):
        if e:
            H[i, e - 1] = 1e-40j if i % 2 else -1.0
    H[7, flen - 1] = float('nan')
    H[8, :] = 1.0
    assert fp_filter.row_ends(H).tolist() == want


def test_step_norms_of_replaced_templates():
    from gwb200 import fp_filter, pipeline
    rng = np.random.default_rng(6)
    IP = torch.from_numpy(rng.uniform(0.5, 2.0, (3, FLEN)).astype(np.float32)).cuda()
    D = torch.from_numpy((1e-6 * (rng.standard_normal((3, FLEN)) + 1j)).astype(np.complex64)).cuda()
    sw, isw = fp_filter.derive_sw(IP)
    cfg = pipeline.FilterConfig(tile=12, form='f16', cand_cap=1 << 12)
    B = pipeline.Bank(synth.random_bank_c1(24, 5), FLEN, DF, sw, cfg)
    f = torch.arange(FLEN, device='cuda', dtype=torch.float64) * DF
    for i in range(B.M):                       # another family: power laws up to the Nyquist bin
        ph = 2e-4 * (i + 1) * f + i
        H = torch.polar((f + 1.0) ** -0.5, ph)
        H[:B.kmin] = 0
        B.H[i] = H.to(torch.complex64)
    for t, ids in enumerate(B.tiles):
        Ht = B.H[B.row0[t]:B.row0[t] + len(ids)]
        r, A, Vh, worst = fp_filter.svd_tile(Ht, sw, B.kmin, cfg.eps)
        B.svd[t] = dict(r=r, A=A, Vh=Vh, worst=worst, Kp=fp_filter.kp_of(r), Kh=fp_filter.kh_of(r))
    ref = fp_filter.sigma2(B.H, IP, DF, B.kmin)[0].cpu().numpy()
    a0, a1 = 8 * 2048, TLEN - 4 * 2048
    mf = pipeline.MatchedFilter(B, TLEN, a0, a1 - a0, cfg)
    # float64 sums of at most 2^15 positive terms in another order: n 2^-53 of the value
    np.testing.assert_allclose(mf.step(D, IP, isw).cpu().numpy(), ref, rtol=2.0 ** 15 * 2.0 ** -53)
    np.testing.assert_allclose(mf.norms(IP).cpu().numpy(), ref, rtol=2.0 ** 15 * 2.0 ** -53)
