"""The complex GEMM's default launch shapes (one CTA per M block or CTA pairs, the split forms' chunk order) at block counts
and widths on both sides of every line of the rule: exact integer operands, values and first indices exact."""
import pytest
import torch

pytestmark = pytest.mark.gpu

FORMS = {'f16': 0, 'bf16': 1, 'bf16x3': 2, 'f16x2': 6}


@pytest.mark.parametrize('form', list(FORMS))
@pytest.mark.parametrize('M', [1, 128, 129, 300, 384, 600])
@pytest.mark.parametrize('Kh', [32, 48, 64, 112, 128, 144, 192])
def test_default_shapes_exact(form, M, Kh):
    from gwb200 import _lib
    g = torch.Generator('cuda').manual_seed(M + Kh)
    Tn, group = 128 * 37 + 24, 16
    dt = torch.float16 if form.startswith('f16') else torch.bfloat16

    def ints(*shape):
        return torch.randint(-1, 2, shape, generator=g, device='cuda').double()

    ah, al, zh, zl = ints(M, 2 * Kh), ints(M, 2 * Kh) / 4, ints(2 * Kh, Tn), ints(2 * Kh, Tn) / 4
    t16 = [x.to(dt).contiguous() for x in (ah, al, zh, zl)]
    split_a, split_z = form in ('bf16x3', 'f16x2'), form == 'bf16x3'

    def product(a, b):                 # A = [Re | Im], Z = [Re ; Im]
        ar, ai, zr, zi = a[:, :Kh], a[:, Kh:], b[:Kh], b[Kh:]
        return torch.stack([ar @ zr - ai @ zi, ai @ zr + ar @ zi])

    z = product(ah, zh)
    if split_a:
        z += product(al, zh)
    if split_z:
        z += product(ah, zl)
    p = (z ** 2).sum(0)                # at most 2 (2 Kh 1.5)^2 in units of 1 / 16: exact in float32
    nout = -(-Tn // (128 * group))
    p = torch.nn.functional.pad(p, (0, nout * 128 * group - Tn), value=-1.0).view(M, nout, -1)
    want = p.amax(2)
    first = (p == want[..., None]).to(torch.uint8).argmax(2) + torch.arange(nout, device='cuda') * 128 * group
    V = torch.empty((M, nout), device='cuda')
    I = torch.empty((M, nout), dtype=torch.int32, device='cuda')
    work = torch.empty(_lib.load().gwb_fused_peaks_cplx_work_bytes(M), dtype=torch.uint8, device='cuda')
    q = _lib.ptr
    _lib.call('gwb_fused_peaks_cplx', FORMS[form], q(t16[0]), q(t16[1]) if split_a else None, 2 * Kh, q(t16[2]),
              q(t16[3]) if split_z else None, Tn, M, Kh, Tn, group, q(V), q(I), nout, None, q(work), work.numel(),
              _lib.stream_ptr())
    assert torch.equal(V.double(), want)
    assert torch.equal(I.long(), first)
