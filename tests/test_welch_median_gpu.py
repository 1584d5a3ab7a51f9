"""The register median of the Welch average against numpy's median, bit for bit, for every count around the networks'
sizes, even and odd, with ties, infinities and NaN frames (whose bins keep the insertion sort's order)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _insertion_median(v):
    """median of the last axis after the insertion sort that leaves an element where nothing before it compares larger"""
    out = np.empty(v.shape[:-1], np.float32)
    for i in np.ndindex(out.shape):
        u = []
        for t in v[i]:
            j = len(u)
            while j > 0 and u[j - 1] > t:
                j -= 1
            u.insert(j, t)
        n = len(u)
        out[i] = u[n // 2] if n % 2 else (u[n // 2 - 1] + u[n // 2]) / np.float32(2)
    return out


@pytest.mark.parametrize('nfr', [1, 2, 3, 15, 16, 17, 31, 32, 33, 62, 63, 64, 65])
def test_median_matches_sorting(nfr):
    from gwb200 import _lib
    rng = np.random.default_rng(nfr)
    rows, nbin, dt, fac, bias = 3, 70, np.float32(0.5), np.float32(1.5), 1.25
    X = (rng.standard_normal((rows, nfr, nbin)) + 1j * rng.standard_normal((rows, nfr, nbin))).astype(np.complex64)
    X[0, :, 5] = X[0, 0, 5]
    X[1, nfr // 2, 6] = np.inf
    X[2, nfr // 3, 7] = np.nan
    re, im = X.real * dt, X.imag * dt
    p = re * re + im * im
    p[:, :, 0] /= 2
    p[:, :, -1] /= 2
    ref = (_insertion_median(p.transpose(0, 2, 1)) / np.float32(bias)) * fac
    Xd = torch.from_numpy(X).cuda()
    psd = torch.empty((rows, nbin), dtype=torch.float32, device='cuda')
    _lib.call('gwb_welch_avg', _lib.ptr(Xd), nbin, rows, nfr, nbin, float(dt), 1, bias, float(fac), _lib.ptr(psd), nbin,
              _lib.stream_ptr())
    assert np.array_equal(psd.cpu().numpy(), ref, equal_nan=True)
