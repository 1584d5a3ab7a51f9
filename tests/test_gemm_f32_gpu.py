"""The packed fp32 GEMM at the edges of its tiles: rows around 64, K around 16 and not a multiple of 4 (4-byte copies),
ragged and misaligned samples, windows shared out over clusters of 1, 2 and 4 CTAs with short last windows. It adds in
the same order with the same rounding as the synchronous kernel, so the two agree bit for bit, first index included."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('M,K,Tn,group,shift', [(1, 1, 1, 1, 0), (63, 16, 128 * 5, 1, 0), (64, 17, 1000, 4, 0),
                                                (65, 68, 128 * 37 + 1, 8, 0), (130, 3, 128 * 33, 7, 1),
                                                (200, 64, 128 * 50 + 64, 16, 0), (40, 36, 128 * 9, 16, 3)])
def test_packed_kernel_equals_the_synchronous_one(M, K, Tn, group, shift):
    from gwb200 import _lib, fp_gemm
    g = torch.Generator(device='cuda').manual_seed(M + K)
    Are, Aim = (torch.randn((M, K), generator=g, device='cuda') for _ in range(2))
    Z = torch.randn((K, Tn + shift), generator=g, device='cuda')[:, shift:]
    Z[:, Tn // 2:Tn // 2 + 200] = Z[:, :1]             # ties: equal columns, the first index wins
    out = {}
    try:
        for on in (1, 0):
            _lib.call('gwb_f32_set_async', on)
            out[on] = fp_gemm.fused_peaks(Are, Aim, Z, M, Tn, group=group)
            torch.cuda.synchronize()
    finally:
        _lib.call('gwb_f32_set_async', 1)
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
