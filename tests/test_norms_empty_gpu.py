"""Norms of no template or no segment are refused by the library's own error."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n,nseg', [(0, 2), (3, 0)])
def test_empty_norms_are_refused(n, nseg):
    from gwb200 import _lib, fp_filter
    with pytest.raises(_lib.GwbError):
        fp_filter.sigma2(torch.zeros((n, 100), dtype=torch.complex64, device='cuda'),
                         torch.zeros((nseg, 100), device='cuda'), 0.1)
