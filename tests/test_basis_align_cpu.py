"""The basis series' C entries refuse buffers that their 16-byte copies cannot read, before any device work: the basis
filters in four-step order from N = 2^19 on, and W wherever the second pass copies it in row chunks."""
import ctypes

import pytest

from gwb200 import _lib


def _series(N, form, **off):
    b = dict.fromkeys(('Vh', 'D', 'tw', 'Vp', 'Dp', 'W', 'Z', 'Zlo', 'partials', 'scale'), 256)
    b.update({k: 256 + v for k, v in off.items()})
    P = ctypes.c_void_p
    return _lib.load().gwb_basis_series(P(b['Vh']), N // 2 + 1, 4, P(b['D']), None, N // 2 + 1, N, P(b['tw']), P(b['Vp']),
                                        P(b['Dp']), P(b['W']), 4, 0, N, form, P(b['Z']), P(b['Zlo']), N, 4,
                                        P(b['partials']), 512, P(b['scale']), None)


def _fused(N, form, **off):
    b = dict.fromkeys(('Vp', 'Dp', 'tw', 'W', 'Z', 'Zlo', 'partials', 'ticket', 'scale'), 256)
    b.update({k: 256 + v for k, v in off.items()})
    P = ctypes.c_void_p
    return _lib.load().gwb_basis_fused(P(b['Vp']), N // 2 + 2, 4, P(b['Dp']), N, P(b['tw']), P(b['W']), 4, 0, N, form,
                                       P(b['Z']), P(b['Zlo']), N, 4, 0, 4, P(b['partials']), 1 << 16, P(b['ticket']),
                                       P(b['scale']), None, None, 0, None)


@pytest.mark.parametrize('log2n,form,buf', [(19, 0, 'Vp'), (20, 1, 'Vp'), (20, 2, 'Vp'), (18, 0, 'W'), (19, 3, 'W'),
                                            (20, 0, 'W'), (20, 2, 'W')])
def test_misaligned_buffers_are_refused(log2n, form, buf):
    for entry in (_series, _fused):
        assert entry(1 << log2n, form, **{buf: 8}) == _lib.GWB_ERR_ALIGN, entry
        assert buf.encode() in _lib.load().gwb_last_error()
