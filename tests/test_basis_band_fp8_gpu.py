"""The banded first pass under the fp8 form, whose row scales come from that pass: same Z bytes and row scales as over the full
band, in one batch of rows and in several, and the same where the data holds a value past the end that is not finite."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('log2n', [19, 20])
@pytest.mark.parametrize('runs', [1, 2, 5, 16])
@pytest.mark.parametrize('wrows', [None, 4])
def test_banded_fp8(log2n, runs, wrows):
    from gwb200 import fp_filter
    N, r = 1 << log2n, 11
    kend = min(runs * 32 * (N // 1024) - 3, N // 2 + 1)
    g = torch.Generator(device='cuda').manual_seed(runs)
    V = torch.view_as_complex(torch.randn((r, N // 2 + 1, 2), generator=g, device='cuda'))
    V = V * torch.linspace(0.5, 2.0, r, device='cuda')[:, None]
    V[:, kend:] = 0
    D = torch.view_as_complex(torch.randn((1, N // 2 + 1, 2), generator=g, device='cuda'))
    ws = fp_filter.FusedBasisWorkspace(N, N // 2 + 1, r, wrows=wrows)
    Vp = fp_filter.fourstep_order(V, N)
    bad = torch.empty(1, dtype=torch.int32, device='cuda')
    out = []
    Dp = fp_filter.fourstep_order(D, N, last_bad=bad)[0]
    for kw in ({}, dict(kend=kend, last_bad=bad)):
        Z = torch.zeros((2 * r, N), dtype=torch.uint8, device='cuda')
        fp_filter.basis_series_fused(ws, Vp, Dp, 0, N, Z, form='fp8', **kw)
        out.append((Z & 0x7f | (Z & 0x80) * ((Z & 0x7f) != 0), ws.rowscale.clone()))      # (zeros of either sign)
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    D[0, N // 2 - 1] = float('inf')
    Dp = fp_filter.fourstep_order(D, N, last_bad=bad)[0]
    for kw in ({}, dict(kend=kend, last_bad=bad)):            # NaN everywhere, scales 1 (a row without a positive sum)
        Z.zero_()
        fp_filter.basis_series_fused(ws, Vp, Dp, 0, N, Z, form='fp8', **kw)
        assert ((Z & 0x7f) == 0x7f).all() and (ws.rowscale == 1.0).all()
