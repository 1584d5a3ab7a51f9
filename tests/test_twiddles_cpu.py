"""The closures can be made where no device is (their buffers are then on the host, as their callers'), and the twiddle table
refuses a host device before anything is launched on a host pointer."""
import pytest
import torch

from gwb200 import fp_filter


def test_closures_on_the_host_make_no_table():
    c = fp_filter.make_closures(10, 2049, 4096, torch.ones(2049), 1e-3, dev='cpu')
    assert callable(c.basis_series) and callable(c.svd_tile) and callable(c.stacked_A)


def test_host_device_is_refused():
    with pytest.raises(ValueError):
        fp_filter.twiddles(4096, 'cpu')
