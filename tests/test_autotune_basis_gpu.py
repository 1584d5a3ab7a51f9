"""Tuning the basis series at 2^20 changes its speed only: the choice gives the default's Z and scale bit for bit, leaves the
ring's configuration as it was where no ring is chosen, and is made on filters that end where the bank's do."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import synth

pytestmark = pytest.mark.gpu
N = 1 << 20


def _ring():
    from gwb200 import _lib
    c = (ctypes.c_int * 3)()
    _lib.call('gwb_basis_ring_get_config', *(ctypes.byref(c, 4 * i) for i in range(3)))
    return list(c)


@pytest.mark.parametrize('form,kend', [('f16', 20000), ('bf16x3', None)])
def test_choice_gives_the_default_series(form, kend):
    from gwb200 import _lib, autotune, fp_filter
    r = 20
    _lib.call('gwb_basis_ring_set_config', 2, 2, 0)
    try:
        best, _ = autotune.tune_basis(N, r, form, kend=kend)
        assert best['ring'] or _ring() == [2, 2, 0]
    finally:
        _lib.call('gwb_basis_ring_set_config', 2, 3, 1)
    g = torch.Generator(device='cuda').manual_seed(3)
    Vp = torch.view_as_complex(torch.randn((r, N // 2 + 2, 2), generator=g, device='cuda'))
    Vp = Vp * torch.linspace(1.0, 2.0, r, device='cuda')[:, None]      # rows of unequal power: the scale tells them apart
    Dp = torch.view_as_complex(torch.randn((N // 2 + 2, 2), generator=g, device='cuda'))
    out = []
    for kw in ({}, dict(ring=best['ring'], wrows=best['wrows'])):
        ws = fp_filter.FusedBasisWorkspace(N, N // 2 + 1, r, **kw)
        Z = torch.zeros((2 * r, N), dtype=fp_filter._z_dtype(form), device='cuda')
        Zlo = torch.zeros_like(Z) if form == 'bf16x3' else None
        s = fp_filter.basis_series_fused(ws, Vp, Dp, 0, N, Z, Zlo, form)
        out.append([Z, s.clone()] + ([Zlo] if Zlo is not None else []))
    assert all(torch.equal(a, b) for a, b in zip(*out))


def test_filter_is_tuned_on_its_banks_band(monkeypatch):
    from gwb200 import autotune, fp_filter, pipeline
    tlen = 1 << 16
    flen = tlen // 2 + 1
    IP = torch.from_numpy(np.random.default_rng(6).uniform(0.5, 2.0, (1, flen)).astype(np.float32)).cuda()
    sw, _ = fp_filter.derive_sw(IP)
    cfg = pipeline.FilterConfig(tile=12, form='f32', cand_cap=1 << 12, autotune=True)
    B = pipeline.Bank(synth.random_bank_c1(24, 5), flen, 2048.0 / tlen, sw, cfg)
    seen = []
    real = autotune.tune_basis
    monkeypatch.setattr(autotune, 'tune_basis', lambda *a, **k: seen.append(k['kend']) or real(*a, **k))
    mf = pipeline.MatchedFilter(B, tlen, 16384, 40960, cfg)
    wide = max(range(len(B.svd)), key=lambda t: B.svd[t]['r'])
    assert seen == [mf.kend[wide]] and 0 < seen[0] < flen
