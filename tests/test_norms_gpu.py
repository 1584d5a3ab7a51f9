"""The template-norm kernel at the edges of its tiles: rows around 16 and 64, segments around 8, 16, 32 and 64, ragged
bins and splits, rows that end early (skipped zero chunks), and non-finite inverse PSDs, which reach the norm even where
the template is zero. Reference: float64 numpy; every product is exact in float64, so the sums agree to their rounding
(a few thousand terms of one sign: 1e-12 relative)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n,nseg,flen,kmin', [(1, 1, 4097, 40), (17, 8, 4097, 3), (64, 9, 8193, 0), (65, 16, 2049, 40),
                                              (40, 17, 5000, 77), (70, 33, 3000, 11), (16, 70, 2500, 1)])
def test_sigma2_tiles(n, nseg, flen, kmin):
    from gwb200 import fp_filter
    rng = np.random.default_rng(n * 100 + nseg)
    H = (rng.standard_normal((n, flen)) + 1j * rng.standard_normal((n, flen))).astype(np.complex64)
    for i in range(n):
        H[i, rng.integers(kmin + 1, flen):] = 0
    IP = rng.uniform(0.1, 2.0, (nseg, flen)).astype(np.float32)
    ref = (np.abs(H[:, kmin:].astype(np.complex128)) ** 2) @ IP[:, kmin:].astype(np.float64).T
    sig, norm = fp_filter.sigma2(torch.from_numpy(H).cuda(), torch.from_numpy(IP).cuda(), 0.5, kmin)
    np.testing.assert_allclose(sig.cpu().numpy(), 2.0 * ref, rtol=1e-12)
    np.testing.assert_allclose(norm.cpu().numpy(), 2.0 / np.sqrt(2.0 * ref), rtol=1e-12)


def test_sigma2_non_finite_inverse_psd():
    from gwb200 import fp_filter
    H = np.zeros((20, 1024), np.complex64)
    H[:, 10:100] = 1.0
    IP = np.ones((3, 1024), np.float32)
    IP[1, 900] = np.inf                    # 0 * inf, past every template's end
    IP[2, 50] = np.nan
    sig, _ = fp_filter.sigma2(torch.from_numpy(H).cuda(), torch.from_numpy(IP).cuda(), 1.0, 0)
    s = sig.cpu().numpy()
    assert np.all(s[:, 0] == 360.0) and np.isnan(s[:, 1:]).all()


def _band(H, kmax, IP, df, kmin):
    from gwb200 import _lib
    n, nseg = H.shape[0], IP.shape[0]
    part = torch.empty(_lib.load().gwb_sigma2_part_elems(n, nseg), dtype=torch.float64, device='cuda')
    sig = torch.empty((n, nseg), dtype=torch.float64, device='cuda')
    _lib.call('gwb_sigma2_band', _lib.ptr(H), H.stride(0), n, _lib.ptr(kmax), _lib.ptr(IP), _lib.row_stride(IP), nseg, kmin,
              H.shape[1], df, _lib.ptr(part), part.numel(), _lib.ptr(sig), nseg, _lib.stream_ptr())
    return sig


@pytest.mark.parametrize('n,nseg,flen,kmin', [(1, 1, 4097, 40), (65, 9, 30001, 3), (130, 33, 9000, 500), (40, 70, 5000, 0)])
def test_sigma2_of_rows_with_ends(n, nseg, flen, kmin):
    rng = np.random.default_rng(n + nseg)
    H = (rng.standard_normal((n, flen)) + 1j * rng.standard_normal((n, flen))).astype(np.complex64)
    kmax = rng.integers(kmin + 1, flen, n).astype(np.int32)
    kmax[n // 2] = kmin                                          # a row of zeros
    for i in range(n):
        H[i, kmax[i]:] = 0
    IP = rng.uniform(0.1, 2.0, (nseg, flen)).astype(np.float32)
    Hd, kd, IPd = torch.from_numpy(H).cuda(), torch.from_numpy(kmax).cuda(), torch.from_numpy(IP).cuda()
    ref = 2.0 * (np.abs(H[:, kmin:].astype(np.complex128)) ** 2) @ IP[:, kmin:].astype(np.float64).T
    np.testing.assert_allclose(_band(Hd, kd, IPd, 0.5, kmin).cpu().numpy(), ref, rtol=1e-12)
    IPd[nseg - 1, flen - 1] = float('inf')                       # past every end: 0 * inf
    s = _band(Hd, kd, IPd, 0.5, kmin).cpu().numpy()
    assert np.isnan(s[:, nseg - 1]).all()
    np.testing.assert_allclose(s[:, :nseg - 1], ref[:, :nseg - 1], rtol=1e-12)
