"""Basis filters that end below the Nyquist bin: the banded first pass gives the full one's Z for every run count (ends on
and around the runs' edges) and both lengths that have one, a non-finite datum past the end makes every output NaN in
both, and the ordering kernel finds the filters' and the data's ends."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(log2n, r, kend, seed=0):
    g = torch.Generator(device='cuda').manual_seed(seed)
    flen = (1 << log2n) // 2 + 1
    V = torch.view_as_complex(torch.randn((r, flen, 2), generator=g, device='cuda'))
    V[:, kend:] = 0
    return V, torch.view_as_complex(torch.randn((flen, 2), generator=g, device='cuda'))


@pytest.mark.parametrize('log2n', [19, 20])
@pytest.mark.parametrize('runs,off', [(1, 0), (1, 1), (2, 0), (3, -5), (4, 0), (7, 100), (8, 0), (8, 1), (16, 0)])
@pytest.mark.parametrize('form', ['f32', 'bf16x3'])
def test_banded_pass_equals_the_full_one(log2n, runs, off, form):
    from gwb200 import fp_filter
    N, r = 1 << log2n, 11
    n2 = N // 1024
    kend = min(runs * 32 * n2 + off, N // 2 + 1)          # a run is 32 k1 of n2 bins
    V, D = _inputs(log2n, r, kend)
    last = torch.empty(1, dtype=torch.int32, device='cuda')
    bad = torch.empty(1, dtype=torch.int32, device='cuda')
    Vp, Dp = fp_filter.fourstep_order(V, N, last_nz=last), fp_filter.fourstep_order(D[None], N, last_bad=bad)[0]
    assert int(last) == kend - 1 and int(bad) == -1
    a0, Tn = 1000, N - 3000
    ws = fp_filter.FusedBasisWorkspace(N, N // 2 + 1, r)
    out = []
    for kw in ({}, dict(kend=kend, last_bad=bad)):
        Z = torch.full((2 * r, Tn), 3.0, dtype=fp_filter._z_dtype(form), device='cuda')
        Zlo = torch.full_like(Z, 5.0) if form == 'bf16x3' else None
        s = fp_filter.basis_series_fused(ws, Vp, Dp, a0, Tn, Z, Zlo, form, **kw)
        out.append([Z, s.clone()] + ([Zlo] if Zlo is not None else []))
    assert all(torch.equal(x, y) for x, y in zip(*out))


@pytest.mark.parametrize('value', [float('inf'), float('nan')])
def test_non_finite_data_past_the_end(value):
    from gwb200 import fp_filter
    N, r, kend = 1 << 19, 9, 5000
    V, D = _inputs(19, r, kend)
    D[200001] = value
    bad = torch.empty(1, dtype=torch.int32, device='cuda')
    Vp, Dp = fp_filter.fourstep_order(V, N), fp_filter.fourstep_order(D[None], N, last_bad=bad)[0]
    assert int(bad) == 200001
    ws = fp_filter.FusedBasisWorkspace(N, N // 2 + 1, r)
    for kw in ({}, dict(kend=kend, last_bad=bad)):
        Z = torch.zeros((2 * r, N), dtype=torch.float32, device='cuda')
        fp_filter.basis_series_fused(ws, Vp, Dp, 0, N, Z, form='f32', **kw)
        assert torch.isnan(Z).all()
