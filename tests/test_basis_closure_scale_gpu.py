"""The drop-in series' scale is summed in float64 from the squares on: data scaled by a power of two far beyond the square
root of float32's range gives the same Z, bit for bit, and the scale times that power; and the scale is the float64 rms
of the float32 samples to the rounding of its own float32."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(log2n, r, a0, Tn, form, p):
    from gwb200 import fp_filter
    N = 1 << log2n
    flen = N // 2 + 1
    g = torch.Generator(device='cuda').manual_seed(log2n + r)
    V = torch.view_as_complex(torch.randn((r, flen, 2), generator=g, device='cuda')) / flen ** 0.5
    D = torch.view_as_complex(torch.randn((flen, 2), generator=g, device='cuda')) * 2.0 ** p
    return fp_filter.make_closures(10, flen, N, torch.ones(flen, device='cuda'), 1e-3, form=form).basis_series(V, D, a0, Tn)


@pytest.mark.parametrize('log2n,r,a0,Tn', [(13, 3, 100, 7777), (16, 9, 8, 60000), (18, 5, 1001, 200003),
                                           (19, 2, 32768, 400000), (20, 9, 77, 1000001)])
def test_power_of_two_scaling(log2n, r, a0, Tn):
    Z, s = _run(log2n, r, a0, Tn, 'f32', 0)
    # Z s are the samples again, each off by at most 2^-24 from Z's rounding and 2^-24 from 1 / s's; the scale is itself
    # rounded to float32
    ref = (Z[:2 * r].double() * s).square().mean().sqrt().item()
    assert abs(s - ref) <= 3 * 2.0 ** -24 * ref
    for p in (-75, 70):
        Zp, sp = _run(log2n, r, a0, Tn, 'f32', p)
        assert sp == s * 2.0 ** p
        assert torch.equal(Zp, Z)
