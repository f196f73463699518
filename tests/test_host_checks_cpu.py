"""Checks of the host side that no GPU is needed for: plane sizes, per-device tables, scratch sizes, threads."""

import ctypes as C
import threading

import pytest
import torch

from turboquant_b200 import _engine as E, _lib


@pytest.mark.parametrize("d,kb,vb", [(128, 3, 2), (256, 4, 4)])
def test_planes_are_measured_before_a_kernel_reads_them(d, kb, vb):
    consts = E.LayerConstants(d, kb, vb, "cpu")
    lay, n = consts.layout, 5
    byte = lambda *s: torch.zeros(*s, dtype=torch.uint8)  # noqa: E731
    codes, signs, norms, rnorms = byte(n, lay.kcode_row), byte(n, lay.ksign_row), torch.ones(n), torch.ones(n, dtype=torch.float16)
    assert E.key_planes_fit(consts, n, codes, signs, norms, rnorms)
    assert E.key_planes_fit(consts, n, codes, None, norms, None)
    for bad in ((codes[:, 1:], signs, norms, rnorms), (codes.int(), signs, norms, rnorms), (codes, signs[:4], norms, rnorms),
                (codes, signs, norms[:4], rnorms), (codes, signs, norms, rnorms[:4]), (codes, signs, norms.double(), rnorms),
                (codes, None, norms, rnorms), (codes, signs, norms, None), (codes, signs, norms.to("meta"), rnorms),
                (byte(lay.kcode_row, n).T, signs, norms, rnorms)):
        assert not E.key_planes_fit(consts, n, *bad)
    data, scales, zeros = byte(n, d * vb // 8), torch.ones(n, d // 32), torch.zeros(n, d // 32)
    assert E.value_planes_fit(n, d, vb, data, scales, zeros)
    for bad in ((data[:4], scales, zeros), (data.int(), scales, zeros), (data, scales[:, 1:], zeros), (data, scales, zeros[:4]),
                (data, scales, zeros.half()), (data, scales.double(), zeros.double()), (data, scales.to("meta"), zeros)):
        assert not E.value_planes_fit(n, d, vb, *bad)
