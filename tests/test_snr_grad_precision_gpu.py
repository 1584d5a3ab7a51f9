"""The float64 gradient kernel's phase, amplitude and norm against extended precision (80-bit), one bin at a time: data that
is one in a single bin gives z = 4 df f^(-7/6) exp(i (Psi(f) - pi / 4)).
Bounds, u = 2^-53, S the sum of the phase's terms in absolute value. A term is a constant, a power of pi Ms and a power of f:
pi Ms carries some 7 u (its pow 4, three products), its -5/3 power 5/3 of that, cube root (2 u), square, product, division
and the polynomial some 13 u more, f^(-5/3) 8 u, the sum of ten terms 3 u, the reduction by 2 pi 1 u: at most 40 u S if all of
them peak together, and, as about twenty independent roundings of rms 0.6 times their bound, 8 u S in the mean square. The
amplitude: sqrt, division, cube root (1 u of its 2), products, the complex product and |z|: 8 u. The norm: 4 u a weight,
and a sum of 1e4 positive terms whose roundings are of either sign: 16 u.
Gradients per component against central differences of the 80-bit form (relative step 1e-8, which turns the phase by
1e-4 rad at most: truncation 1e-8, rounding 1e-10): 2e-5 of the component and 1e-7 of the largest; in the float32 form, whose
products and phases are rounded to 24 bits, 1e-3 and 1e-4."""
import numpy as np
import pytest
import torch

from oracle import adjoint as oa
from oracle import synth

pytestmark = pytest.mark.gpu
L = np.longdouble
U = 2.0 ** -53
PI = L(3.141592653589793)
TWO_PI = L('6.283185307179586476925286766559005768')


def phase80(mc, q, c1, c2, e0, f, f_ecc=10.0):
    """(Psi(f), sum of its terms' absolute values) in 80-bit arithmetic."""
    mc, q, c1, c2, e0 = (L(x) for x in (mc, q, c1, c2, e0))
    eta = q / (1 + q) ** 2
    X = PI * L(4.925490947641267e-06) * mc * np.power(eta, L(-3) / 5)
    v = np.power(X * f, L(1) / 3)
    d1, d2 = 1 / (1 + q), q / (1 + q)
    beta = L(113) / 12 * (d1 * d1 * c1 + d2 * d2 * c2) + L(6.25) * eta * (c1 + c2)
    sigma = L(474) / 48 * eta * c1 * c2
    lv, l6, l4 = np.log(v), -np.log(L(6)) / 2, np.log(L(4))
    p5 = PI * (L(38645) / 756 - L(65) / 9 * eta)
    p6 = (L(11583231236531) / L(4694215680) - L(640) / 3 * PI * PI - L(6848) / 21 * L(0.5772156649015329)
          + (L(-15737765635) / 3048192 + L(2255) / 12 * PI * PI) * eta + L(76055) / 1728 * eta ** 2
          - L(127825) / 1296 * eta ** 3)
    terms = [1 + 0 * f, v ** 2 * L(20) / 9 * (L(743) / 336 + L(11) / 4 * eta), v ** 3 * -16 * PI, v ** 3 * 4 * beta,
             v ** 4 * 10 * (L(3058673) / 7257600 + L(5429) / 1008 * eta + L(617) / 144 * eta ** 2),
             v ** 4 * -10 * sigma, v ** 5 * p5, v ** 5 * p5 * 3 * (lv - l6), v ** 6 * p6, v ** 6 * L(-6848) / 21 * (lv + l4),
             v ** 7 * PI * (L(77096675) / 254016 + L(378515) / 1512 * eta - L(74045) / 756 * eta ** 2),
             L(-2355) / 1462 * e0 * e0 * np.power(L(f_ecc) / f, L(19) / 9)]
    pre = L(3) / 128 / eta / v ** 5
    return pre * sum(terms), pre * sum(abs(t) for t in terms)


@pytest.mark.parametrize('seed,lo,hi', [(0, 1.2, 3.0), (1, 3.0, 9.0), (2, 9.0, 40.0)])
def test_phase_and_amplitude_per_bin(seed, lo, hi):
    from gwb200 import adjoint
    n, flen, df = 2048, 16385, 2048.0 / 32768
    kmin = int(20.0 / df)
    rng = np.random.default_rng(seed)
    th = np.zeros((n, 7))
    th[:, 0] = np.exp(rng.uniform(np.log(lo), np.log(hi), n))
    th[:, 1] = rng.uniform(0.3, 1.0, n)
    th[:, 2:4] = rng.uniform(-0.9, 0.9, (n, 2))
    th[:, 4] = np.where(rng.random(n) < 0.5, rng.uniform(0.05, 0.3, n), 0.0)
    kend = np.array([oa.kmax(m, q, df, flen) for m, q in th[:, :2]])
    k = np.where(np.arange(n) % 2 == 0, kmin, (kmin * (kend / kmin) ** rng.random(n)).astype(int))
    k = np.minimum(np.maximum(k, kmin), kend - 1)
    D = torch.zeros((n, flen), dtype=torch.complex64, device='cuda')
    D[torch.arange(n), torch.from_numpy(k)] = 1.0
    IP = torch.ones(flen, device='cuda')
    r = adjoint.snr_grad(torch.from_numpy(th).cuda(), D, IP, df, kmin, fp64=True)
    z = r['z'].cpu().numpy()
    f = k.astype(L) * L(df)
    psi, S = phase80(*th[:, :5].T, f)
    ref = psi - PI / 4
    d = np.angle(z).astype(L) - (ref - TWO_PI * np.rint(ref / TWO_PI))
    d = (d - TWO_PI * np.rint(d / TWO_PI)).astype(float)
    e = d / (U * S.astype(float))
    assert np.abs(e).max() <= 40.0, np.abs(e).max()
    assert np.sqrt(np.mean(e[::2] ** 2)) <= 8.0 and np.sqrt(np.mean(e[1::2] ** 2)) <= 8.0, \
        (np.sqrt(np.mean(e[::2] ** 2)), np.sqrt(np.mean(e[1::2] ** 2)))
    amp = 4 * L(df) * np.power(f, L(-7) / 6)
    assert np.abs((np.abs(z.astype(np.clongdouble)) - amp) / amp).max() <= 8 * U
    w = np.power(np.arange(flen, dtype=L)[kmin:] * L(df), L(-7) / 3)
    cs = np.concatenate([[L(0)], np.cumsum(w)])
    sig = 4 * L(df) * cs[kend - kmin]
    assert np.abs((r['sigma2'].cpu().numpy().astype(L) - sig) / sig).max() <= 16 * U


@pytest.mark.parametrize('mc,nb,log2n', [(25.0, 16, 15), (5.0, 16, 15), (9.0, 32, 14), (1.3, 16, 15), (30.0, 2, 16)])
@pytest.mark.parametrize('fp64', [True, False])
def test_gradients_per_component(mc, nb, log2n, fp64):
    from gwb200 import adjoint
    N, sr = 1 << log2n, 2048.0
    flen, df = N // 2 + 1, sr / N
    kmin = int(20.0 / df)
    rng = np.random.default_rng(nb + log2n)
    f = np.arange(flen) * df
    IP = np.zeros(flen, np.float32)
    IP[kmin:] = 1.0 / synth.analytic_psd(f[kmin:])
    th = np.array([mc, 0.7, 0.3, -0.2, 0.1, 0.5 * N / sr, 1.0])
    h, _ = oa.template(th + np.array([1e-3 * mc / (1 + 40 * (mc < 2)), 0, 0, 0, 0, 1e-4, 0]), flen, df, kmin)
    a = 15.0 / np.sqrt(4 * df * np.sum(np.abs(h) ** 2 * IP))
    noise = (rng.standard_normal(flen) + 1j * rng.standard_normal(flen)) / np.sqrt(4 * df * np.maximum(IP, 1e-30))
    D = ((a * h + noise * (IP > 0)) * IP).astype(np.complex64)
    r = adjoint.snr_grad(torch.from_numpy(th[None].copy()).cuda(), torch.from_numpy(D[None].copy()).cuda(), torch.from_numpy(IP).cuda(),
                         df, kmin, nbins=nb, fp64=fp64)
    # central differences with the phase in 80 bits (the band's end and the bins do not move in the step)
    k1 = oa.kmax(th[0], th[1], df, flen)
    e = oa.edges(IP, df, kmin, k1, nb)
    fb = np.arange(kmin, k1).astype(L) * L(df)
    w = 4 * L(df) * np.power(fb, L(-7) / 6) * D[kmin:k1].astype(np.clongdouble)
    sig2 = 4 * L(df) * np.sum(np.power(fb, L(-7) / 3) * IP[kmin:k1].astype(L))

    def stats(t):
        ph = phase80(*t[:5], fb)[0] - PI / 4 + 2 * PI * fb * L(t[5]) - L(t[6])
        ph = ph - TWO_PI * np.rint(ph / TWO_PI)
        q = w * (np.cos(ph) + 1j * np.sin(ph))
        zj = np.array([q[e[j] - kmin:e[j + 1] - kmin].sum() for j in range(nb)])
        z = abs(zj.sum())
        snr, chisq = z / np.sqrt(sig2), (nb * np.sum(np.abs(zj) ** 2) - z ** 2) / sig2
        rc = chisq / (2 * nb - 2)
        return np.array([snr, chisq, snr if rc <= 1 else snr / ((1 + rc ** 3) / 2) ** (L(1) / 6)])

    g = np.zeros((3, 7))
    for p, scale in enumerate((1.0, 1.0, 1.0, 1.0, 0.1, 1e-3, 1.0)):
        step = 1e-8 * max(abs(th[p]), scale) if p != 5 else 1e-9
        up, dn = th.astype(L), th.astype(L)
        up[p] += L(step)
        dn[p] -= L(step)
        g[:, p] = ((stats(up) - stats(dn)) / (up[p] - dn[p])).astype(float)
    for row, name in enumerate(('dsnr', 'dchisq', 'dnewsnr')):
        got, want = r[name][0].cpu().numpy(), g[row]
        tol = (2e-5, 1e-7) if fp64 else (1e-3, 1e-4)
        assert np.all(np.abs(got - want) <= tol[0] * np.abs(want) + tol[1] * np.abs(want).max()), (name, got, want)
