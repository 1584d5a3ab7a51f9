"""The first pass's band limit goes with the last bad bins of the very data it reads: a caller's own ordered data, set or
written after a step on other data, gives the series that it gives in a fresh filter object."""
import numpy as np
import pytest
import torch

from oracle import synth

pytestmark = pytest.mark.gpu

TLEN = 1 << 19                                   # the shortest transform whose first pass stops at the filters' end
FLEN = TLEN // 2 + 1
DF = 2048.0 / TLEN
A0, TN = 32768, 425984


def _setup():
    from gwb200 import fp_filter, pipeline
    rng = np.random.default_rng(8)
    IP = torch.from_numpy(rng.uniform(0.5, 2.0, (1, FLEN)).astype(np.float32)).cuda()
    good = torch.from_numpy((1e-6 * (rng.standard_normal((1, FLEN)) + 1j)).astype(np.complex64)).cuda()
    bad = good.clone()
    bad[0, FLEN - 5] = float('inf')
    sw, isw = fp_filter.derive_sw(IP)
    cfg = pipeline.FilterConfig(tile=6, form='f32', cand_cap=1 << 14)
    B = pipeline.Bank(synth.random_bank_c1(6, 5), FLEN, DF, sw, cfg)
    mf = pipeline.MatchedFilter(B, TLEN, A0, TN, cfg)
    assert max(mf.kend) < FLEN - 5
    return fp_filter, mf, good, bad, IP, isw


def _series(mf, D, IP, isw):
    sig = mf.norms(IP)
    mf.counters.zero_()
    mf.tile_segment(0, D, isw, sig, 0)
    r = mf.bank.svd[0]['r']
    return mf.Z[:r].clone()


@pytest.mark.parametrize('how', ['set', 'set_first', 'write'])
def test_band_limit_follows_the_data(how):
    fp_filter, mf, good, bad, IP, isw = _setup()
    want = {}
    for name, D in (('good', good), ('bad', bad)):
        mf.order_data(D, isw)
        want[name] = _series(mf, D, IP, isw)
    assert torch.isfinite(want['good']).all() and torch.isnan(want['bad']).all()
    for last, now, D in ((good, 'bad', bad), (bad, 'good', good)):
        if how == 'set_first':
            fp_filter, mf, *_ = _setup()
            mf.Dp = fp_filter.fourstep_order(last, TLEN, isw)
        mf.step(last, IP, isw)
        if how == 'write':
            fp_filter.fourstep_order(D, TLEN, isw, out=mf.Dp)
        else:
            mf.Dp = fp_filter.fourstep_order(D, TLEN, isw)
        got = _series(mf, D, IP, isw)
        # the band's limit changes no bits but the signs of zeros
        assert torch.equal(torch.nan_to_num(got, nan=7.0), torch.nan_to_num(want[now], nan=7.0)), (how, now)
    # and a step after that pairs them again
    mf.step(bad, IP, isw)
    assert torch.isnan(mf.Z[:mf.bank.svd[0]['r']]).all()
