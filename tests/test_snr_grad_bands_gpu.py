"""The gradient kernel's values over its band lengths and bin counts: bands that fit the kept table and longer ones,
bands cut unevenly by the warps, 1, 2, 16 and 32 chi-squared bins. float64 form against the float64 oracle: sums of at
most 1e4 terms whose phases (up to 1e4 rad) are good to 1e-11, so 1e-9; the gradients against its central differences
(relative step 1e-6: 1e-4 of the largest)."""
import numpy as np
import pytest
import torch

from oracle import adjoint as oa
from oracle import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('mc,nb,log2n', [(25.0, 16, 15), (5.0, 16, 15), (9.0, 32, 14), (12.0, 1, 15), (30.0, 2, 16)])
def test_values_and_gradients(mc, nb, log2n):
    from gwb200 import adjoint
    N, sr = 1 << log2n, 2048.0
    flen, df = N // 2 + 1, sr / N
    kmin = int(20.0 / df)
    rng = np.random.default_rng(nb + log2n)
    f = np.arange(flen) * df
    IP = np.zeros(flen, np.float32)
    IP[kmin:] = 1.0 / synth.analytic_psd(f[kmin:])
    th = np.array([[mc, 0.7, 0.3, -0.2, 0.1, 0.5 * N / sr, 1.0], [mc * 1.1, 0.9, 0.0, 0.0, 0.0, 0.4 * N / sr, 0.2]])
    D = np.zeros((2, flen), np.complex64)
    for i in range(2):
        h, _ = oa.template(th[i] + np.array([1e-3 * mc, 0, 0, 0, 0, 1e-4, 0]), flen, df, kmin)
        a = 15.0 / np.sqrt(4 * df * np.sum(np.abs(h) ** 2 * IP))
        n = (rng.standard_normal(flen) + 1j * rng.standard_normal(flen)) / np.sqrt(4 * df * np.maximum(IP, 1e-30))
        D[i] = ((a * h + n * (IP > 0)) * IP).astype(np.complex64)
    r = adjoint.snr_grad(torch.from_numpy(th).cuda(), torch.from_numpy(D).cuda(), torch.from_numpy(IP).cuda(), df, kmin,
                         nbins=nb, fp64=True)
    for i in range(2):
        if nb > 1:
            snr, chisq, ns = oa.snr_chisq(th[i], D[i], IP, df, kmin, nb)
            np.testing.assert_allclose([r['snr'][i].item(), r['chisq'][i].item(), r['newsnr'][i].item()],
                                       [snr, chisq, ns], rtol=1e-9)
            g = oa.fd_grad(th[i], D[i], IP, df, kmin, nb)
            for k, row in (('dsnr', 0), ('dchisq', 1)):
                got = r[k][i].cpu().numpy()
                assert np.abs(got - g[row]).max() <= 1e-4 * np.abs(g[row]).max() + 1e-6, (k, got, g[row])
        else:
            q = 4 * df * np.conj(oa.template(th[i], flen, df, kmin)[0]) * D[i].astype(np.complex128)
            assert abs(complex(r['z'][i].item()) - q.sum()) <= 1e-9 * abs(q.sum())
