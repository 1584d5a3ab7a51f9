"""The reference-layout basis series through the fused passes: every transform length's kernels, one to more than a
batch of rows, spans that cut a pass's blocks, each Z encoding, against a float64 transform. Tolerances: the scale is an
rms of more than 1e4 float32 sums (1e-6 relative); Z within its type's rounding of z / scale plus 1e-5 of the rms."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
EPS = {'f16': 2.0 ** -11, 'f32': 0.0, 'bf16': 2.0 ** -8, 'bf16x3': 2.0 ** -16}


@pytest.mark.parametrize('log2n,r,a0,Tn,form', [(12, 1, 0, 4096, 'f32'), (13, 65, 100, 7777, 'f16'),
                                                (15, 3, 4097, 20000, 'bf16x3'), (16, 70, 8, 60000, 'bf16'),
                                                (18, 5, 1001, 200003, 'f16'), (19, 2, 32768, 400000, 'f32'),
                                                (20, 66, 98304, 917504, 'f16'), (20, 9, 77, 1000001, 'f32')])
def test_series_matches_float64(log2n, r, a0, Tn, form):
    from gwb200 import fp_filter
    N = 1 << log2n
    flen = N // 2 + 1
    g = torch.Generator(device='cuda').manual_seed(log2n * 100 + r)
    V = torch.view_as_complex(torch.randn((r, flen, 2), generator=g, device='cuda')) / flen ** 0.5
    D = torch.view_as_complex(torch.randn((flen, 2), generator=g, device='cuda'))
    c = fp_filter.make_closures(10, flen, N, torch.ones(flen, device='cuda'), 1e-3, form=form)
    Z, scale = c.basis_series(V, D, a0, Tn)
    Z = Z[0].double() + Z[1].double() if form == 'bf16x3' else Z.double()
    assert Z.shape[0] % 64 == 0 and not Z[2 * r:].any()
    z = torch.empty((r, Tn), dtype=torch.complex128, device='cuda')
    for j in range(r):
        q = torch.zeros(N, dtype=torch.complex128, device='cuda')
        q[:flen] = V[j].to(torch.complex128).conj() * D.to(torch.complex128)
        z[j] = torch.fft.ifft(q, norm='forward')[a0:a0 + Tn]
    ref = torch.view_as_real(z[:64]).square().mean().sqrt().item()
    assert abs(scale - ref) <= 1e-6 * ref
    for got, want in ((Z[:r], z.real / scale), (Z[r:2 * r], z.imag / scale)):
        assert ((got - want).abs() <= EPS[form] * want.abs() + 1e-5).all()
