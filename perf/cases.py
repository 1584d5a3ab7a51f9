"""Performance cases of the framework: what its users have it do, through the public entry points, with the sizes of its
configurations, tests and benchmark. `listed` names the fixed cases, `draw` gives more of the same ranges; `prepare`
makes the inputs and what a user's program keeps (bank, plan, workspace), `run` is one pass, `work` counts the bytes and
operations that a pass cannot do without and `exact` computes the outputs in 64 bits with plain torch.

Inputs: coloured Gaussian noise of the analytic PSD (scaled strain units), TaylorF2 chirps in it, banks of TaylorF2
templates of the two synthetic mass ranges, and Gaussian operands where an entry point takes plain matrices."""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'gw-gpu-search_b200')
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

SR = 2048.0
F_LOW = 20.0
NBINS = 16
MTSUN = 4.925490947641267e-06
DYN2 = 5.9029581035870565e+20 ** 2
PEAK_ROWS = 8192
BANK = 5880                     # templates of the production-scale bank; its tiles hold 256 of them in chirp-time order


def listed():
    return [
        # the smallest call: peaks of a few windows of a short dense series, where the launch counts
        dict(name='peaks_small', kind='peaks', rows=8, n=16384, a0=512, cw=2048, nwin=7),
        # the reference-layout fp16 GEMM with block maxima, at its autotuner's default shape
        dict(name='gemm_f16', kind='gemm', form='f16', M=1024, K=128, Tn=1 << 20, group=1),
        # the split-bf16 GEMM on stacked operands: one tile of 256 templates against a 512 s chunk, 1 s windows
        dict(name='gemm_split', kind='gemm', form='bf16x3', M=256, K=64, Tn=917504, group=16),
        # the plain fp32 GEMM, a ragged number of rows (the bank's last tile) and of samples
        dict(name='gemm_f32', kind='gemm', form='f32', M=248, K=192, Tn=458700, group=16),
        # the reference's basis-series closure (float scale back, fp16 Z), one tile against a 512 s chunk
        dict(name='basis_closure', kind='closure', form='f16', r=100, log2n=20, a0=98304, Tn=917504, fmax=200.0),
        # the pipeline's fused basis series, one tile against a 512 s chunk
        dict(name='basis_fused', kind='basis', form='f16', r=128, log2n=20, a0=98304, Tn=917504, fmax=200.0),
        # the plain method: 64 non-spinning templates, one 256 s segment, one detector, fp32
        dict(name='step_plain', kind='step', bank='small', n=64, tile=0, log2n=19, nseg=1, form='f32', a0=32768,
             Tn=475136, thr=5.5, ninj=1),
        # the mixed-precision batched filter: one tile of the production bank against four 512 s segments
        dict(name='step_split', kind='step', bank='large', n=256, tile=11, log2n=20, nseg=4, form='bf16x3', a0=98304,
             Tn=917504, thr=6.0, ninj=4),
        # the exact stage of one (tile, segment): z, bin power and edges at its candidates
        dict(name='exact_peaks', kind='exact', n=256, log2n=20, npeaks=320),
        # SNR, newSNR and chi-squared of 16 s triggers with their gradients over seven parameters
        dict(name='gradients', kind='grad', n=2048, log2n=15, fp64=False, shared=False),
        # conditioning (median Welch PSD, truncation, D and 1/PSD) of a batch of 512 s chunks
        dict(name='condition', kind='condition', nds=16, log2n=20),
        # float64 template norms of one tile against a batch of segments
        dict(name='norms', kind='norms', n=256, nseg=16, log2n=20),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['peaks', 'gemm', 'gemm', 'closure', 'basis', 'step', 'step', 'exact', 'grad', 'condition',
                       'norms'])
    if kind == 'peaks':
        cw, nwin = rng.choice([256, 1024, 2048, 3000]), _log(rng, 2, 192)
        a0 = rng.randrange(0, 4097)
        return dict(kind=kind, rows=_log(rng, 1, 64), n=a0 + cw * nwin + rng.randrange(0, 999), a0=a0, cw=cw, nwin=nwin)
    if kind == 'gemm':
        form = rng.choice(['f16', 'bf16x3', 'f32'])
        # row strides of the 16-bit operands are 16-byte aligned for TMA: their lengths are multiples of 8 samples
        Tn = _log(rng, 1 << 14, 1 << 19)
        if form != 'f32':
            Tn = Tn // 8 * 8
        K = 64 if form == 'bf16x3' else rng.choice([64, 128])
        return dict(kind=kind, form=form, M=_log(rng, 16, 512), K=K if form != 'f32' else K + rng.choice([0, 4, 64]),
                    Tn=Tn, group=rng.choice([1, 8, 16]))
    if kind in ('closure', 'basis'):
        p = rng.randrange(16, 21)
        N = 1 << p
        Tn = (N * rng.randrange(12, 15) // 16) // 2048 * 2048
        a0 = rng.randrange(0, (N - Tn) // 2 + 1) // 8 * 8
        return dict(kind=kind, form=rng.choice(['f16', 'f32'] if kind == 'closure' else ['f16', 'f32', 'bf16']),
                    r=_log(rng, 12, 100), log2n=p, a0=a0, Tn=Tn, fmax=float(rng.randrange(60, 900)))
    if kind == 'step':
        p = rng.randrange(17, 20)
        N = 1 << p
        Tn = (N * 13 // 16) // 2048 * 2048
        large = rng.random() < 0.6
        return dict(kind=kind, bank='large' if large else 'small', n=rng.randrange(24, 193), tile=rng.randrange(0, 23),
                    log2n=p, nseg=rng.randrange(1, 4), form=rng.choice(['bf16x3', 'bf16x3', 'f32']),
                    a0=N // 16, Tn=Tn, thr=6.0, ninj=2)
    if kind == 'exact':
        return dict(kind=kind, n=rng.randrange(24, 257), log2n=rng.randrange(17, 21), npeaks=_log(rng, 8, 800))
    if kind == 'grad':
        return dict(kind=kind, n=_log(rng, 16, 1500), log2n=rng.choice([14, 15, 15]), fp64=rng.random() < 0.4,
                    shared=rng.random() < 0.5)
    if kind == 'condition':
        return dict(kind=kind, nds=rng.randrange(1, 13), log2n=rng.randrange(18, 21))
    return dict(kind=kind, n=rng.randrange(20, 257), nseg=rng.randrange(1, 17), log2n=rng.randrange(17, 21))


# ---- the physics of the inputs, in float64 torch -------------------------------------------------------------------

def _psd(f):
    """Analytic broadband detector PSD in scaled units, flat below 15 Hz at a high wall."""
    x = f.clamp(min=15.0) / 215.0
    s = 1e-49 * (x ** -4.14 - 5.0 * x ** -2 + 111.0 * (1.0 - x ** 2 + 0.5 * x ** 4) / (1.0 + 0.5 * x ** 2))
    return torch.where(f < 15.0, 1e4 * s, s) * DYN2


def _phase(f, m1, m2, c1, c2, e0, f_ecc=10.0):
    """TaylorF2 phase to 3.5PN with aligned-spin terms and the leading eccentric term; f_ISCO in the logarithm."""
    M = m1 + m2
    eta = m1 * m2 / M ** 2
    ms = math.pi * MTSUN * M
    v = (ms * f) ** (1.0 / 3.0)
    beta = (113.0 / 12.0) * ((m1 / M) ** 2 * c1 + (m2 / M) ** 2 * c2) + 6.25 * eta * (c1 + c2)
    sigma = eta * (474.0 / 48.0) * c1 * c2
    g, pi = 0.5772156649015329, math.pi
    p2 = 20.0 / 9.0 * (743.0 / 336.0 + 11.0 / 4.0 * eta)
    p3 = -16.0 * pi + 4.0 * beta
    p4 = 10.0 * (3058673.0 / 7257600.0 + 5429.0 / 1008.0 * eta + 617.0 / 144.0 * eta ** 2) - 10.0 * sigma
    p5 = pi * (38645.0 / 756.0 - 65.0 / 9.0 * eta) * (1.0 + 3.0 * torch.log(v * math.sqrt(6.0)))
    p6 = (11583231236531.0 / 4694215680.0 - 640.0 / 3.0 * pi ** 2 - 6848.0 / 21.0 * g
          + eta * (-15737765635.0 / 3048192.0 + 2255.0 / 12.0 * pi ** 2) + 76055.0 / 1728.0 * eta ** 2
          - 127825.0 / 1296.0 * eta ** 3 - 6848.0 / 21.0 * torch.log(4.0 * v))
    p7 = pi * (77096675.0 / 254016.0 + 378515.0 / 1512.0 * eta - 74045.0 / 756.0 * eta ** 2)
    s = 1.0 + v * v * (p2 + v * (p3 + v * (p4 + v * (p5 + v * (p6 + v * p7)))))
    v0 = (ms * f_ecc) ** (1.0 / 3.0)
    s = s - 2355.0 / 1462.0 * e0 ** 2 * (v0 / v) ** (19.0 / 3.0)
    return 3.0 / (128.0 * eta * v ** 5) * s


def _kend(m1, m2, df, flen):
    """Exclusive end bin of a template: the bin after f_ISCO, at most the last but one."""
    f = 1.0 / (6.0 ** 1.5 * math.pi * (m1 + m2) * MTSUN)
    return torch.clamp(torch.floor(f / df) + 1, max=flen - 1).to(torch.int64)


def _chirps(b, flen, df):
    """(n, flen) complex128 templates f^-7/6 exp(-i (Psi - pi/4)) on [20 Hz, f_ISCO] and their end bins."""
    kmin = int(F_LOW / df)
    k1 = _kend(b['mass1'], b['mass2'], df, flen)
    H = torch.zeros((len(k1), flen), dtype=torch.complex128, device='cuda')
    top = int(k1.max())
    f = torch.arange(kmin, top, device='cuda', dtype=torch.float64) * df
    for r in range(0, len(k1), 32):
        c = [b[k][r:r + 32, None] for k in ('mass1', 'mass2', 'spin1z', 'spin2z', 'ecc')]
        h = torch.polar(f ** (-7.0 / 6.0), f * 0) * torch.polar(torch.ones_like(f), -(_phase(f, *c) - math.pi / 4))
        on = torch.arange(kmin, top, device='cuda') < k1[r:r + 32, None]
        H[r:r + 32, kmin:top] = torch.where(on, h, torch.zeros_like(h))
    return H, k1


def _bank(case, seed):
    """Templates of one tile: non-spinning of 5-50 solar masses ('small'), or the chosen 256-wide tile of the 5,880
    aligned-spin and eccentric ones of 3-100 solar masses in chirp-time order ('large'). numpy arrays."""
    rng = np.random.default_rng([seed, 17])
    if case.get('bank', 'large') == 'small':
        m = np.sort(rng.uniform(5.0, 50.0, (case['n'], 2)), axis=1)
        z = np.zeros(case['n'])
        return dict(mass1=m[:, 1], mass2=m[:, 0], spin1z=z, spin2z=z, ecc=z)
    na, ne = 4612, BANK - 4612
    m = np.sort(rng.uniform(3.0, 100.0, (na, 2)), axis=1)
    mt, q = rng.uniform(45.0, 100.0, ne), rng.uniform(1.0, 3.0, ne)
    z = np.zeros
    b = dict(mass1=np.r_[m[:, 1], mt * q / (1 + q)], mass2=np.r_[m[:, 0], mt / (1 + q)],
             spin1z=np.r_[rng.uniform(-0.9, 0.9, na), z(ne)], spin2z=np.r_[rng.uniform(-0.9, 0.9, na), z(ne)],
             ecc=np.r_[z(na), rng.uniform(0.0, 0.3, ne)])
    mc = (b['mass1'] * b['mass2']) ** 0.6 / (b['mass1'] + b['mass2']) ** 0.2
    order = np.argsort(mc ** (-5.0 / 3.0), kind='stable')          # chirp time goes with Mc^(-5/3)
    first = min(case.get('tile', 0) * 256, BANK - case['n'])
    ids = order[first:first + case['n']]
    return {k: v[ids] for k, v in b.items()}


def _gen(seed):
    return torch.Generator(device='cuda').manual_seed(int(seed))


def _cnormal(shape, g, dtype=torch.float32):
    return torch.view_as_complex(torch.randn(tuple(shape) + (2,), generator=g, device='cuda', dtype=dtype))


def _noise(rows, flen, df, g, kmin):
    """Noise spectra (complex128) and inverse PSDs (float64) of `rows` segments, whose levels differ by a few percent."""
    f = torch.arange(flen, device='cuda', dtype=torch.float64) * df
    level = 1.0 + 0.05 * torch.randn((rows, 1), generator=g, device='cuda', dtype=torch.float64).clamp(-3, 3)
    psd = _psd(f) * level
    ip = 1.0 / psd
    ip[:, :kmin] = 0.0
    return _cnormal((rows, flen), g).to(torch.complex128) * torch.sqrt(psd / (4.0 * df)), ip


# ---- kinds of case: inputs, one pass, 64-bit outputs ---------------------------------------------------------------

def prepare(case, seed):
    return globals()['_prepare_' + case['kind']](case, seed)


def run(s):
    return globals()['_run_' + s['kind']](s)


def exact(case, seed):
    return globals()['_exact_' + case['kind']](case, seed)


def _peaks_in(case, seed):
    return _cnormal((case['rows'], case['n']), _gen(seed))


def _prepare_peaks(case, seed):
    from gwb200 import peak_kernel  # noqa: F401
    return dict(case, z=_peaks_in(case, seed))


def _run_peaks(s):
    from gwb200 import peak_kernel
    return peak_kernel.window_peaks(s['z'], s['a0'], s['cw'], s['nwin'])


def _exact_peaks(case, seed):
    z = _peaks_in(case, seed)[:, case['a0']:case['a0'] + case['cw'] * case['nwin']].to(torch.complex128)
    p = (z.real ** 2 + z.imag ** 2).reshape(case['rows'], case['nwin'], case['cw'])
    return p.amax(2), None


def _gemm_in(case, seed):
    """Stacked operands Are = [Re, -Im], Aim = [Im, Re] (M x K) of unit-norm rows and Z (K x Tn) of unit variance."""
    g = _gen(seed)
    M, K, Tn = case['M'], case['K'], case['Tn']
    a = torch.randn((M, K), generator=g, device='cuda') / math.sqrt(K)
    re, im = a[:, :K // 2], a[:, K // 2:]
    ops = [torch.cat([re, -im], 1), torch.cat([im, re], 1), torch.randn((K, Tn), generator=g, device='cuda')]
    if case['form'] == 'f16':
        return [x.half() for x in ops]
    if case['form'] == 'bf16x3':
        hi = [x.bfloat16() for x in ops]
        return [t for x, h in zip(ops, hi) for t in (h, (x - h.float()).bfloat16())]
    return ops


def _prepare_gemm(case, seed):
    from gwb200 import fp_gemm  # noqa: F401
    return dict(case, ops=_gemm_in(case, seed))


def _run_gemm(s):
    from gwb200 import fp_gemm
    if s['form'] == 'bf16x3':
        return fp_gemm.fused_peaks_split(*s['ops'], s['M'], s['Tn'], group=s['group'])
    return fp_gemm.fused_peaks(*s['ops'], s['M'], s['Tn'], group=s['group'])


def _exact_gemm(case, seed):
    ops = [t.double() if t.shape[0] == case['M'] else t for t in _gemm_in(case, seed)]
    if case['form'] == 'bf16x3':
        ops = [ops[0] + ops[1], ops[2] + ops[3], (ops[4], ops[5])]
    else:
        ops = [ops[0], ops[1], (ops[2],)]
    w = 128 * case['group']
    out = []
    step = max(1, (1 << 17) // w) * w
    for t in range(0, case['Tn'], step):
        z = sum(x[:, t:t + step].double() for x in ops[2])
        p = (ops[0] @ z) ** 2 + (ops[1] @ z) ** 2
        n = p.shape[1]
        p = torch.nn.functional.pad(p, (0, -n % w), value=-1.0)
        out.append(p.reshape(p.shape[0], -1, w).amax(2))
    return torch.cat(out, 1), None


def _series_in(case, seed):
    """Basis filters (r, flen) on [20 Hz, fmax), unit norm over the band, and one segment's whitened data."""
    g = _gen(seed)
    N = 1 << case['log2n']
    flen, df = N // 2 + 1, SR / N
    kmin, k1 = int(F_LOW / df), min(int(case['fmax'] / df), flen - 1)
    Vh = torch.zeros((case['r'], flen), dtype=torch.complex64, device='cuda')
    amp = (torch.arange(kmin, k1, device='cuda') * df) ** (-7.0 / 6.0)
    Vh[:, kmin:k1] = _cnormal((case['r'], k1 - kmin), g) * (amp / amp.norm())
    D = _cnormal((flen,), g)
    D[:kmin] = 0
    return N, flen, kmin, Vh, D


def _prepare_closure(case, seed):
    from gwb200 import fp_filter
    N, flen, kmin, Vh, D = _series_in(case, seed)
    sw = torch.ones(flen, dtype=torch.float32, device='cuda')
    return dict(case, c=fp_filter.make_closures(kmin, flen, N, sw, 1e-3, form=case['form']), Vh=Vh, D=D)


def _run_closure(s):
    return s['c'].basis_series(s['Vh'], s['D'], s['a0'], s['Tn'])


def _series64(case, seed):
    N, flen, kmin, Vh, D = _series_in(case, seed)
    r = case['r']
    z = torch.empty((r, case['Tn']), dtype=torch.complex128, device='cuda')
    power = torch.empty(r, dtype=torch.float64, device='cuda')
    for j in range(0, r, 16):
        q = torch.zeros((min(16, r - j), N), dtype=torch.complex128, device='cuda')
        q[:, :flen] = Vh[j:j + 16].to(torch.complex128).conj() * D.to(torch.complex128)
        x = torch.fft.ifft(q, norm='forward')
        power[j:j + 16] = (x.real ** 2 + x.imag ** 2).mean(1)
        z[j:j + 16] = x[:, case['a0']:case['a0'] + case['Tn']]
    return z, power


def _exact_closure(case, seed):
    z, _ = _series64(case, seed)
    r = case['r']
    first = torch.view_as_real(z[:64])
    scale = float(first.square().mean().sqrt())
    Z = torch.zeros((-(-2 * r // 64) * 64, case['Tn']), dtype=torch.float64, device='cuda')
    Z[:r], Z[r:2 * r] = z.real / scale, z.imag / scale
    return Z, scale


def _prepare_basis(case, seed):
    from gwb200 import fp_filter
    N, flen, kmin, Vh, D = _series_in(case, seed)
    dt = {'f16': torch.float16, 'f32': torch.float32, 'bf16': torch.bfloat16}[case['form']]
    return dict(case, ws=fp_filter.FusedBasisWorkspace(N, flen, case['r']), Vp=fp_filter.fourstep_order(Vh, N),
                Dp=fp_filter.fourstep_order(D, N), Z=torch.zeros((2 * case['r'], case['Tn']), dtype=dt, device='cuda'))


def _run_basis(s):
    from gwb200 import fp_filter
    scale = fp_filter.basis_series_fused(s['ws'], s['Vp'], s['Dp'], s['a0'], s['Tn'], s['Z'], form=s['form'])
    return s['Z'], scale


def _exact_basis(case, seed):
    z, power = _series64(case, seed)
    # the scale is the rms of one component over the whole series of the first rows: two of them at 2^20, else 64
    scale = torch.sqrt(power[:2 if case['log2n'] == 20 else 64].mean() / 2.0)
    return torch.cat([z.real, z.imag]) / scale, scale[None]


def _segments(case, seed, bank):
    """Data spectra with injected chirps of the bank, and inverse PSDs: (nseg, flen) complex128 and float64."""
    N = 1 << case['log2n']
    flen, df = N // 2 + 1, SR / N
    kmin = int(F_LOW / df)
    X, ip = _noise(case['nseg'], flen, df, _gen(seed), kmin)
    rng = np.random.default_rng([seed, 23])
    ids = rng.integers(0, case['n'], case['ninj'])
    h, _ = _chirps({k: torch.from_numpy(v[ids]).cuda() for k, v in bank.items()}, flen, df)
    f = torch.arange(flen, device='cuda', dtype=torch.float64) * df
    for i in range(case['ninj']):
        s = i % case['nseg']
        t0 = (case['a0'] + rng.uniform(0.1, 0.9) * case['Tn']) / SR
        hi = h[i] * torch.polar(torch.ones_like(f), -2.0 * math.pi * f * t0)
        snr = torch.sqrt(4.0 * df * (hi.abs() ** 2 * ip[s]).sum())
        X[s] += rng.uniform(12.0, 24.0) / snr * hi
    return X, ip


def _prepare_step(case, seed):
    from gwb200 import fp_filter, pipeline
    N = 1 << case['log2n']
    flen, df = N // 2 + 1, SR / N
    bank = _bank(case, seed)
    X, ip = _segments(case, seed, bank)
    D, IP = (X * ip).to(torch.complex64), ip.to(torch.float32)
    sw, isw = fp_filter.derive_sw(IP)
    cfg = pipeline.FilterConfig(tile=256, form=case['form'], snr_threshold=case['thr'], nbins=NBINS, cand_cap=1 << 15)
    B = pipeline.Bank(bank, flen, df, sw, cfg)
    mf = pipeline.MatchedFilter(B, N, case['a0'], case['Tn'], cfg)
    return dict(case, mf=mf, D=D, IP=IP, isw=isw)


def _run_step(s):
    mf = s['mf']
    sig = mf.step(s['D'], s['IP'], s['isw'])
    r = mf.results()
    c, p = r['cands'], r['peaks']
    o = np.lexsort((c['window'], c['seg'], c['row']))     # the peak table's order: template, then time
    table = dict(row=c['row'], seg=c['seg'], window=c['window'], snr=p['snr'], chisq=p['chisq'])
    out = dict(sigma2=sig, window_max=mf.V)
    for k, v in table.items():
        out[k] = np.zeros(PEAK_ROWS, v.dtype)              # a table of fixed length, zero past the last peak
        out[k][:len(o)] = v[o]
    return out


def _exact_step(case, seed):
    N = 1 << case['log2n']
    flen, df = N // 2 + 1, SR / N
    bank = _bank(case, seed)
    X, ip = _segments(case, seed, bank)
    mc = (bank['mass1'] * bank['mass2']) ** 0.6 / (bank['mass1'] + bank['mass2']) ** 0.2
    bank = {k: v[np.argsort(mc ** (-5.0 / 3.0), kind='stable')] for k, v in bank.items()}
    H, _ = _chirps({k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in bank.items()}, flen, df)
    sig = 4.0 * df * (H.real ** 2 + H.imag ** 2) @ ip.T
    # the window maxima that remain after a step are the last segment's
    D = X[-1] * ip[-1]
    nw = case['Tn'] // 2048
    V = torch.empty((case['n'], nw), dtype=torch.float64, device='cuda')
    for r in range(0, case['n'], 16):
        q = torch.zeros((min(16, case['n'] - r), N), dtype=torch.complex128, device='cuda')
        q[:, :flen] = H[r:r + 16].conj() * D
        z = torch.fft.ifft(q, norm='forward')[:, case['a0']:case['a0'] + nw * 2048]
        p = (z.real ** 2 + z.imag ** 2) * (16.0 * df * df / sig[r:r + 16, -1:])
        V[r:r + 16] = p.reshape(p.shape[0], nw, 2048).amax(2)
    # the candidates' own values hang on which samples the filter chose
    return dict(sigma2=sig, window_max=V, row=None, seg=None, window=None, snr=None, chisq=None)


def _exact_in(case, seed):
    N = 1 << case['log2n']
    flen, df = N // 2 + 1, SR / N
    kmin = int(F_LOW / df)
    b = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in _bank(dict(n=case['n'], tile=6), seed).items()}
    H, k1 = _chirps(b, flen, df)
    X, ip = _noise(1, flen, df, _gen(seed), kmin)
    rng = np.random.default_rng([seed, 29])
    rows = rng.integers(0, case['n'], case['npeaks'])
    samples = rng.integers(N // 16, N - N // 16, case['npeaks'])
    return (N, df, kmin, H.to(torch.complex64), k1.cpu().numpy(), (X[0] * ip[0]).to(torch.complex64),
            ip[0].to(torch.float32), rows, samples)


def _prepare_exact(case, seed):
    from gwb200 import exact_stage
    N, df, kmin, H, k1, D, IP, rows, samples = _exact_in(case, seed)
    tile = exact_stage.TemplateTile(H, np.full(case['n'], NBINS), kmin, k1)
    return dict(case, stage=exact_stage.ExactStage(tile), seg=exact_stage.SegmentData(D, IP, df, N), rows=rows,
                samples=samples)


def _run_exact(s):
    from gwb200 import exact_stage
    v = s['stage'].evaluate(s['seg'], exact_stage.PeakRequest(s['rows'], s['samples']))
    return v.z, v.pw, v.fpeak


def _exact_exact(case, seed):
    N, df, kmin, H, k1, D, IP, rows, samples = _exact_in(case, seed)
    z, pw, fp = [], [], []
    for r, t in zip(rows.tolist(), samples.tolist()):
        h = H[r, kmin:int(k1[r])].to(torch.complex128)
        k = torch.arange(kmin, int(k1[r]), device='cuda')
        cs = torch.cumsum((h.real ** 2 + h.imag ** 2) * IP[kmin:int(k1[r])].double(), 0)
        frac = torch.arange(1, NBINS, device='cuda', dtype=torch.float64) / NBINS
        e = torch.searchsorted(cs / cs[-1], frac, right=True)
        j = torch.zeros(len(k), dtype=torch.int64, device='cuda')
        j[e] = 1 if len(torch.unique(e)) == len(e) else torch.bincount(e, minlength=len(k))[e]
        a = 2.0 * math.pi / N * ((k * t) % N).double()
        q = h.conj() * D[kmin:int(k1[r])].to(torch.complex128) * torch.polar(torch.ones_like(a), a)
        zj = torch.zeros((NBINS, 2), dtype=torch.float64, device='cuda')
        zj.index_add_(0, torch.cumsum(j, 0), torch.view_as_real(q))
        z.append(torch.complex(zj[:, 0].sum(), zj[:, 1].sum()))
        pw.append(zj.square().sum())
        fp.append((2.0 * (int(e[-1]) + kmin) - (int(e[-2]) + kmin)) * df)
    return torch.stack(z), torch.stack(pw), np.array(fp)


def _grad_in(case, seed):
    """Triggers of the production bank's parameters: data holding a chirp of SNR 8-40, parameters near its own."""
    N = 1 << case['log2n']
    n, flen, df = case['n'], N // 2 + 1, SR / N
    kmin = int(F_LOW / df)
    rng = np.random.default_rng([seed, 31])
    ecc = rng.random(n) < 0.22
    m = np.sort(rng.uniform(5.0, 40.0, (n, 2)), axis=1)
    b = dict(mass1=m[:, 1], mass2=m[:, 0], spin1z=np.where(ecc, 0, rng.uniform(-0.9, 0.9, n)),
             spin2z=np.where(ecc, 0, rng.uniform(-0.9, 0.9, n)), ecc=np.where(ecc, rng.uniform(0.05, 0.3, n), 0.0))
    tc = rng.uniform(0.4, 0.6, n) * N / SR
    X, ip = _noise(n, flen, df, _gen(seed), kmin)
    if case['shared']:
        X, ip = X * torch.sqrt(ip[:, -1:] / ip[:1, -1:]), ip[:1]
    h, _ = _chirps({k: torch.from_numpy(v).cuda() for k, v in b.items()}, flen, df)
    f = torch.arange(flen, device='cuda', dtype=torch.float64) * df
    h = h * torch.polar(torch.ones_like(f), -2.0 * math.pi * f * torch.from_numpy(tc).cuda()[:, None])
    snr = torch.sqrt(4.0 * df * (h.abs() ** 2 * ip).sum(1, keepdim=True))
    D = (X + torch.from_numpy(rng.uniform(8.0, 40.0, (n, 1))).cuda() / snr * h) * ip
    mc = (b['mass1'] * b['mass2']) ** 0.6 / (b['mass1'] + b['mass2']) ** 0.2
    th = np.stack([mc * (1 + rng.normal(0, 2e-3, n)), b['mass2'] / b['mass1'], b['spin1z'], b['spin2z'], b['ecc'],
                   tc + rng.normal(0, 2e-4, n), rng.uniform(0, 6.28, n)], 1)
    ip = ip[0] if case['shared'] else ip
    return torch.from_numpy(th).cuda(), D.to(torch.complex64), ip.to(torch.float32), df, kmin


_GRAD = ('snr', 'newsnr', 'chisq', 'sigma2', 'dsnr', 'dnewsnr', 'dchisq')


def _prepare_grad(case, seed):
    from gwb200 import adjoint  # noqa: F401
    th, D, IP, df, kmin = _grad_in(case, seed)
    return dict(case, th=th, D=D, IP=IP, df=df, kmin=kmin)


def _run_grad(s):
    from gwb200 import adjoint
    r = adjoint.snr_grad(s['th'], s['D'], s['IP'], s['df'], s['kmin'], nbins=NBINS, fp64=s['fp64'])
    # sums of the fp32 form are float32 values in the float64 table: kept as such, as a trigger table does
    return {k: r[k] if s['fp64'] else r[k].float() for k in _GRAD}


def _exact_grad(case, seed):
    th, D, IP, df, kmin = _grad_in(case, seed)
    out = {k: [] for k in _GRAD}
    flen = D.shape[1]
    for i in range(0, case['n'], 64):
        t = th[i:i + 64].clone().requires_grad_(True)
        mc, q, c1, c2, e0, tc, pc = [t[:, p:p + 1] for p in range(7)]
        m1 = mc * (q / (1 + q) ** 2) ** -0.6 / (1 + q)
        k1 = _kend(m1.detach(), (q * m1).detach(), df, flen)
        k = torch.arange(kmin, int(k1.max()), device='cuda')
        on, f = k < k1, k.double() * df
        ip = (IP if IP.dim() == 1 else IP[i:i + 64])[..., kmin:int(k1.max())].double()
        d = D[i:i + 64, kmin:int(k1.max())].to(torch.complex128)
        amp = torch.where(on, f ** (-7.0 / 6.0), torch.zeros_like(d.real))
        w = amp ** 2 * ip
        cs = torch.cumsum(w, 1)
        tot = w.sum(1)
        j = sum((cs > b / NBINS * cs[:, -1:]).to(torch.int64) for b in range(1, NBINS))
        ph = _phase(f, m1, q * m1, c1, c2, e0) - math.pi / 4 + 2 * math.pi * f * tc - pc
        co, si = torch.cos(ph) * amp, torch.sin(ph) * amp
        z0 = torch.zeros((len(t), NBINS), dtype=torch.float64, device='cuda')
        zr = 4 * df * z0.scatter_add(1, j, co * d.real - si * d.imag)
        zi = 4 * df * z0.scatter_add(1, j, co * d.imag + si * d.real)
        sig2 = 4 * df * tot
        z2 = zr.sum(1) ** 2 + zi.sum(1) ** 2
        snr = torch.sqrt(z2 / sig2)
        chisq = (NBINS * (zr ** 2 + zi ** 2).sum(1) - z2) / sig2
        rc = chisq / (2 * NBINS - 2)
        ns = torch.where(rc > 1, snr * ((1 + rc.clamp(min=1) ** 3) / 2) ** (-1.0 / 6.0), snr)
        for name, v in (('snr', snr), ('newsnr', ns), ('chisq', chisq)):
            out[name].append(v.detach())
            out['d' + name].append(torch.autograd.grad(v.sum(), t, retain_graph=True)[0])
        out['sigma2'].append(sig2)
    return {k: torch.cat(v) for k, v in out.items()}


def _strain(case, seed):
    """(nds, n) float32 strain: coloured noise."""
    N = 1 << case['log2n']
    f = torch.arange(N // 2 + 1, device='cuda', dtype=torch.float64) * (SR / N)
    X = _cnormal((case['nds'], N // 2 + 1), _gen(seed)) * torch.sqrt(_psd(f) * N * SR / 4.0).to(torch.float32)
    X[:, 0] = 0
    return torch.fft.irfft(X.to(torch.complex64), n=N).contiguous()


def _prepare_condition(case, seed):
    from gwb200 import gpu_prep
    N = 1 << case['log2n']
    return dict(case, x=_strain(case, seed),
                cond=gpu_prep.BatchConditioner(case['nds'], N, SR, F_LOW, 16.0, 8.0, N // 16384 - 1, 16.0))


def _run_condition(s):
    return s['cond'](s['x'])


def _exact_condition(case, seed):
    x = _strain(case, seed)
    N, L, st = 1 << case['log2n'], 32768, 16384
    flen, df = N // 2 + 1, SR / N
    kmin, nfr = int(F_LOW / df), N // 16384 - 1
    w = torch.from_numpy(np.hanning(L)).cuda()
    bias = 1.0 + sum(1.0 / (2 * i + 1) - 1.0 / (2 * i) for i in range(1, (nfr - 1) // 2 + 1))
    D, IP = [], []
    for r in range(case['nds']):
        xr = x[r].double()
        p = (torch.fft.rfft(xr.unfold(0, L, st) * w) / SR).abs() ** 2
        p[:, 0] /= 2
        p[:, -1] /= 2
        p = torch.sort(p, 0).values
        med = 0.5 * (p[(nfr - 1) // 2] + p[nfr // 2]) / bias * (2.0 * SR / (w * w).sum())
        k = torch.arange(flen, device='cuda', dtype=torch.float64) * (L / N)
        lo = k.floor().clamp(max=L // 2 - 1).to(torch.int64)
        psd = med[lo] + (med[lo + 1] - med[lo]) * (k - lo)
        inv = torch.zeros(flen, dtype=torch.complex128, device='cuda')
        inv[kmin:N // 2] = 1.0 / torch.sqrt(psd[kmin:N // 2])
        q = torch.fft.irfft(inv, n=N, norm='forward') * df
        q[L // 2:N - L // 2] = 0.0
        ip = (torch.fft.rfft(q) / (df * N)).abs() ** 2
        ip[:kmin] = 0.0
        D.append(torch.fft.rfft(xr) / SR * ip)
        IP.append(ip)
    return torch.stack(D), torch.stack(IP)


def _norms_in(case, seed):
    N = 1 << case['log2n']
    flen, df = N // 2 + 1, SR / N
    b = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda()
         for k, v in _bank(dict(n=case['n'], tile=6), seed).items()}
    H, _ = _chirps(b, flen, df)
    _, ip = _noise(case['nseg'], flen, df, _gen(seed), int(F_LOW / df))
    return H.to(torch.complex64), ip.to(torch.float32), df


def _prepare_norms(case, seed):
    from gwb200 import fp_filter  # noqa: F401
    H, IP, df = _norms_in(case, seed)
    return dict(case, H=H, IP=IP, df=df, kmin=int(F_LOW / df))


def _run_norms(s):
    from gwb200 import fp_filter
    return fp_filter.sigma2(s['H'], s['IP'], s['df'], s['kmin'])


def _exact_norms(case, seed):
    H, IP, df = _norms_in(case, seed)
    h = H.to(torch.complex128)
    sig = 4.0 * df * (h.real ** 2 + h.imag ** 2) @ IP.double().T
    return sig, 4.0 * df / torch.sqrt(sig)


# ---- what a pass cannot do without ---------------------------------------------------------------------------------

def work(case):
    kind = case['kind']
    N = 1 << case.get('log2n', 0)
    flen = N // 2 + 1
    fft = 5.0 * N * max(1, case.get('log2n', 1))
    if kind == 'peaks':
        n = case['rows'] * case['nwin']
        return dict(bytes=n * (case['cw'] * 8 + 8), flops=3.0 * n * case['cw'])
    if kind == 'gemm':
        M, K, Tn = case['M'], case['K'], case['Tn']
        es = 2 if case['form'] == 'f16' else 4
        nout = -(-(-(-Tn // 128)) // case['group'])
        return dict(bytes=es * (2 * M * K + K * Tn) + 8 * M * nout,
                    flops=4.0 * M * K * Tn * (3 if case['form'] == 'bf16x3' else 1))
    if kind in ('closure', 'basis'):
        es = 4 if case['form'] == 'f32' else 2
        return dict(bytes=8 * (case['r'] + 1) * flen + 2 * case['r'] * case['Tn'] * es, flops=case['r'] * (fft + 3 * N))
    if kind == 'step':
        # the basis keeps about half as many rows as a tile has templates
        n, S, r = case['n'], case['nseg'], (case['n'] + 1) // 2
        p = 3 if case['form'] == 'bf16x3' else 1
        return dict(bytes=8 * (n + r) * flen + 12 * S * flen + 8 * n * S + 8 * n * (case['Tn'] // 2048) * S,
                    flops=S * (8.0 * p * n * r * case['Tn'] + r * fft + 2.0 * n * flen))
    if kind == 'exact':
        rows = min(case['n'], case['npeaks'])
        return dict(bytes=8 * (rows + 1) * flen + 4 * flen, flops=8.0 * case['npeaks'] * flen)
    if kind == 'grad':
        return dict(bytes=case['n'] * flen * (8 if case['shared'] else 12) + case['n'] * 280,
                    flops=100.0 * case['n'] * flen)
    if kind == 'condition':
        return dict(bytes=case['nds'] * (4 * N + 12 * flen), flops=case['nds'] * 2.5 * fft)
    return dict(bytes=8 * case['n'] * flen + 4 * case['nseg'] * flen + 8 * case['n'] * case['nseg'],
                flops=2.0 * case['n'] * case['nseg'] * flen + 3.0 * case['n'] * flen)
