"""Default workspace of the basis series at 2^20: W is bounded however many rows there are, and the rows' batches and the ring
leave no trace in Z."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('rows', [1, 2, 700])
def test_default_workspace(rows):
    from gwb200 import fp_filter
    N = 1 << 20
    g = torch.Generator(device='cuda').manual_seed(rows)
    Vp = torch.view_as_complex(torch.randn((rows, N // 2 + 2, 2), generator=g, device='cuda'))
    Dp = torch.view_as_complex(torch.randn((N // 2 + 2, 2), generator=g, device='cuda'))
    a0, Tn = 4096, 65536
    out = []
    for kw in ({}, dict(wrows=rows), dict(ring=True)):
        ws = fp_filter.FusedBasisWorkspace(N, N // 2 + 1, rows, **kw)
        if not kw:
            assert ws.W.shape[0] == min(rows, 640)
        Z = torch.zeros((2 * rows, Tn), dtype=torch.float16, device='cuda')
        s = fp_filter.basis_series_fused(ws, Vp, Dp, a0, Tn, Z, form='f16')
        out.append((Z, s.clone()))
        del ws
    for Z, s in out[1:]:
        assert torch.equal(Z, out[0][0]) and torch.equal(s, out[0][1])
