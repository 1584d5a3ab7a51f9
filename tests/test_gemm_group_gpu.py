"""Output groups larger than the row, up to the largest int: one output per row, as with a group of exactly its blocks."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('form', ['f32', 'f16', 'bf16x3'])
@pytest.mark.parametrize('group', [38, 39, 2 ** 30, 2 ** 31 - 1])
def test_group_beyond_the_row(form, group):
    from gwb200 import fp_gemm
    g = torch.Generator('cuda').manual_seed(group % 1000)
    M, K, Tn = 70, 64, 128 * 37 + 8                       # 38 blocks of 128 samples
    A = [torch.randint(-3, 4, (M, K), generator=g, device='cuda').float() for _ in range(2)]
    Z = torch.randint(-3, 4, (K, Tn), generator=g, device='cuda').float()
    p = (A[0] @ Z) ** 2 + (A[1] @ Z) ** 2                 # integers below 2^24: exact
    if form == 'bf16x3':
        b = [x.bfloat16() for x in (*A, Z)]
        zero = [torch.zeros_like(x) for x in b]
        V, I = fp_gemm.fused_peaks_split(b[0], zero[0], b[1], zero[1], b[2], zero[2], M, Tn, group=group)
    else:
        dt = torch.float32 if form == 'f32' else torch.float16
        V, I = fp_gemm.fused_peaks(A[0].to(dt), A[1].to(dt), Z.to(dt), M, Tn, group=group)
    assert V.shape == (M, 1)
    assert torch.equal(V[:, 0].double(), p.amax(1).double())
    assert torch.equal(I[:, 0].long(), (p == p.amax(1, keepdim=True)).to(torch.uint8).argmax(1))
