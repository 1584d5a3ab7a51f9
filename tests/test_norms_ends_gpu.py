"""Template norms of a bank whose chi-squared bands (kmax) stop before its templates do: whole templates count, in the
filter object and in the C step."""
import numpy as np
import pytest
import torch

from oracle import synth

pytestmark = pytest.mark.gpu

TLEN = 1 << 16
FLEN = TLEN // 2 + 1
DF = 2048.0 / TLEN


def test_norms_count_whole_templates():
    from gwb200 import cstep, fp_filter, pipeline
    rng = np.random.default_rng(4)
    IP = torch.from_numpy(rng.uniform(0.5, 2.0, (3, FLEN)).astype(np.float32)).cuda()
    D = torch.from_numpy((1e-6 * (rng.standard_normal((3, FLEN)) + 1j)).astype(np.complex64)).cuda()
    sw, isw = fp_filter.derive_sw(IP)
    cfg = pipeline.FilterConfig(tile=12, form='f16', cand_cap=1 << 12)
    B = pipeline.Bank(synth.random_bank_c1(24, 5), FLEN, DF, sw, cfg)
    B.kmax.copy_(B.kmax // 2)
    ref = fp_filter.sigma2(B.H, IP, DF, B.kmin)[0]
    a0, a1 = 8 * 2048, TLEN - 4 * 2048
    sig = pipeline.MatchedFilter(B, TLEN, a0, a1 - a0, cfg).norms(IP)
    sig_c = cstep.CStep(B, TLEN, a0, a1 - a0, 3, cfg).step(D, IP, isw)
    # float64 sums of at most 2^15 positive terms in another order: n 2^-53 of the value
    for s in (sig, sig_c):
        np.testing.assert_allclose(s.cpu().numpy(), ref.cpu().numpy(), rtol=2.0 ** 15 * 2.0 ** -53)
