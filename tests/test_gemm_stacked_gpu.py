"""The stacked tensor-core GEMM where its work split can go wrong: one and two M blocks, rows past M, one to many windows
per CTA, windows cut between the CTAs of a pair, short last tiles and windows. Small-integer operands, so every sum is
exact and ties are common: maxima and first indices equal the oracle's exactly."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('M,K,Tn,group', [(1, 64, 128, 1), (128, 64, 128 * 9 + 8, 1), (129, 128, 128 * 300, 1),
                                          (100, 64, 128 * 16 * 149 + 40, 16), (256, 64, 128 * 7 * 155, 7),
                                          (300, 128, 128 * 16 * 75, 16), (250, 64, 128 * 3 * 448 - 64, 3)])
@pytest.mark.parametrize('split', [False, True])
def test_work_split(M, K, Tn, group, split):
    from gwb200 import fp_gemm
    if split and K > 64:
        pytest.skip('the split form holds K = 64')
    rng = np.random.default_rng(M + group)
    Are, Aim = (rng.integers(-2, 3, (M, K)).astype(np.float32) for _ in range(2))
    Z = rng.integers(-1, 2, (K, Tn)).astype(np.float32)
    t = lambda a: torch.from_numpy(a).cuda()
    if split:
        z0 = lambda a: torch.zeros_like(t(a)).bfloat16()
        V, I = fp_gemm.fused_peaks_split(t(Are).bfloat16(), z0(Are), t(Aim).bfloat16(), z0(Aim), t(Z).bfloat16(), z0(Z),
                                         M, Tn, group=group)
    else:
        V, I = fp_gemm.fused_peaks(t(Are).half(), t(Aim).half(), t(Z).half(), M, Tn, group=group)
    p = (t(Are) @ t(Z)) ** 2 + (t(Aim) @ t(Z)) ** 2          # exact in float32
    w = 128 * group
    p = torch.nn.functional.pad(p, (0, -Tn % w), value=-1.0).reshape(M, -1, w)
    ref = p.amax(2)
    first = (p == ref[..., None]).to(torch.int8).argmax(2) + w * torch.arange(p.shape[1], device='cuda')
    assert torch.equal(V, ref) and torch.equal(I.long(), first)
