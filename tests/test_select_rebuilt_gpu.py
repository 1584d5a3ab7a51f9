"""Rebuilt complex SNR of the window candidates: the sums over the rows of Z, at lengths around the kernel's steps of 32
elements and rounds of four steps, stacked and compact operands, each form."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('form', [0, 1, 2, 3, 5])
@pytest.mark.parametrize('K,kh', [(64, 0), (200, 0), (64, 32), (192, 96), (256, 128), (320, 160)])
def test_rebuilt_sums(form, K, kh):
    from gwb200 import _exact, _lib
    if form == 5 and kh == 0:
        pytest.skip('the compact layout only')
    n, nw, Tn = 3, 70, 70 * 128
    dt = {0: torch.float16, 1: torch.float32, 2: torch.bfloat16, 3: torch.bfloat16, 5: torch.float16}[form]
    g = torch.Generator('cuda').manual_seed(5 + K + form)

    def operand(*shape):
        x = torch.randn(*shape, device='cuda', generator=g)
        hi = x.to(dt)
        return hi, (x - hi.float()).to(dt)

    (Are, Are_lo), (Aim, Aim_lo), (Z, Zlo) = operand(n, K), operand(n, K), operand(K, Tn)
    V = torch.rand(n, nw, device='cuda', generator=g)
    V[1] = 0.0                                       # a row without candidates
    I = (torch.arange(nw, device='cuda') * 128 + torch.randint(0, 128, (n, nw), device='cuda', generator=g)).int()
    cap = n * nw
    out = {k: torch.zeros(cap * d.itemsize, dtype=torch.uint8, device='cuda')
           for k, d in (('c', _exact.CAND), ('g', _exact.GROUP), ('u', _exact.UNIT))}
    counters = torch.zeros(5, dtype=torch.int32, device='cuda')
    p = _lib.ptr
    _lib.call('gwb_select_windows', p(V), p(I), nw, n, nw, 0.5, 0.0, 0.0, 1000, 0, 0, p(Are), p(Aim), p(Are_lo),
              p(Aim_lo), K, p(Z), p(Zlo), Tn, K, kh, form, None, p(out['c']), cap, p(out['g']), cap, p(out['u']), cap,
              None, 0, p(counters), _lib.stream_ptr())
    nc = int(counters[0])
    assert nc == int((V > 0.5).sum()) > 0 and int(counters[3]) == 0
    c = _exact.from_dev(out['c'], _exact.CAND, nc)
    row, col = torch.tensor(c['row'].astype(np.int64)), torch.tensor(c['sample'].astype(np.int64) - 1000)
    split_a, split_z = form in (2, 5), form == 2
    f = lambda hi, lo, on: (hi.double() + (lo.double() if on else 0.0)).cpu()       # noqa: E731
    zz = f(Z, Zlo, split_z)[:, col].T                                               # (nc, K)
    ar, ai = f(Are, Are_lo, split_a)[row], f(Aim, Aim_lo, split_a)[row]
    if kh:
        wr, wi = ar[:, :kh], ar[:, kh:]
        zr, zs = zz[:, :kh], zz[:, kh:]
        re, im = wr * zr - wi * zs, wi * zr + wr * zs
        absr, absi = (wr * zr).abs() + (wi * zs).abs(), (wi * zr).abs() + (wr * zs).abs()
    else:
        re, im = ar * zz, ai * zz
        absr, absi = re.abs(), im.abs()
    # at most K + 2 roundings of fused steps and 5 of the lanes' sum, and one for each operand's hi + lo
    bound = (K + 9) * 2.0 ** -24
    for got, want, mag in ((c['zr'], re, absr), (c['zi'], im, absi)):
        err = (torch.tensor(got).double() - want.sum(1)).abs()
        assert bool((err <= bound * mag.sum(1)).all())
