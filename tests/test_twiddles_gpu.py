"""One twiddle table per length and device, whichever way the device is named, complete when it is handed out."""
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_one_table_per_device():
    from gwb200 import fp_filter
    N = 1 << 13
    t = fp_filter.twiddles(N)
    i = torch.cuda.current_device()
    assert fp_filter.twiddles(N, 'cuda:%d' % i) is t and fp_filter.twiddles(N, torch.device('cuda', i)) is t


def test_table_is_complete_for_other_streams():
    from gwb200 import fp_filter
    N = 1 << 17
    want = np.exp(2j * np.pi * np.arange(N) / N)
    fp_filter._TWIDDLES.pop((N, torch.cuda.current_device()), None)
    got = []

    def use():
        with torch.cuda.stream(torch.cuda.Stream()):
            got.append(fp_filter.twiddles(N).cpu().numpy())

    ts = [threading.Thread(target=use) for _ in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    # the table's entries are float32 roundings of sin and cos: half a unit each
    for g in got:
        assert np.abs(g.real - want.real).max() <= 2.0 ** -24 and np.abs(g.imag - want.imag).max() <= 2.0 ** -24
