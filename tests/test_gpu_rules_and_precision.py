"""Rules of the dispatch on both sides of their lines, and the precision of the fast paths against 64 bits."""

import math

import pytest
import torch

from oracle import tq_oracle as O
from tests.test_gpu_parity import _bit_frac, _cos, test_prefill_attention_vs_fp32_reference as prefill_against_fp32

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    return torch.device("cuda:0")


def _unpack(packed, width):
    return torch.stack([(packed >> s) & ((1 << width) - 1) for s in range(0, 8, width)], -1).flatten(-2).long()


def _width(bits):
    return 2 if bits == 3 else 4


def _keys64(consts, codes, signs, norms, rnorms):
    """Dequantised keys in 64 bits."""
    y = consts.centroids.double()[_unpack(codes, _width(consts.key_bits))]
    s = _unpack(signs, 1).double() * 2 - 1
    return (y @ consts.Pi.double()) * norms.double()[..., None] + consts.qjl_scale * rnorms.double()[..., None] * (s @ consts.S.double())


def _wrong(consts, x, codes, signs):
    """Codes and sign bits of rows x (n, D) that 64-bit arithmetic on the same rounded unit vectors decides otherwise."""
    norm = x.double().norm(dim=-1).to(x.dtype)
    q = x.double() / (norm.float() + 1e-10).to(x.dtype).double()[:, None]
    rotate = consts.Pi.double().T
    code = torch.searchsorted(consts.boundaries[1:-1].double().contiguous(), (q.float().to(x.dtype).double() @ rotate).contiguous())
    got = _unpack(codes, _width(consts.key_bits))
    r = q @ rotate - consts.centroids.double()[got]
    sign = r @ (consts.S.double() @ rotate).T > 0
    same = (got == code).all(-1)
    return int((got != code).sum()), int((sign != _unpack(signs, 1).bool())[same].sum())


@pytest.mark.parametrize("qh,h,tiles", [(8, 2, 24), (8, 2, 27), (15, 3, 10), (16, 4, 10), (12, 4, 13), (13, 13, 13), (4, 1, 43)])
def test_prefill_on_both_sides_of_the_line_for_pairs(qh, h, tiles, dev):
    """More than a wave of query tiles: single tiles up to the line, pairs beyond it; a ragged last tile."""
    prefill_against_fp32(128, qh, h, tiles * 128 - 37, torch.bfloat16, dev)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_prefill_pairs_are_as_exact_as_single_tiles(dtype, dev):
    """The same heads in one launch (pairs of query tiles) and in eight (single tiles): both round probabilities and
    outputs to 16 bits, so the errors against 64 bits agree; 2e-3 is four times what separates the two here."""
    from turboquant_b200 import _engine as E
    n, qh, h, d = 400, 64, 8, 128
    g = torch.Generator(device=dev)
    g.manual_seed(17)
    q, k, v = (torch.randn(n, x, d, generator=g, device=dev).to(dtype) for x in (qh, h, h))
    pairs = E.prefill_attention(q, k, v)
    single = torch.cat([E.prefill_attention(q[:, 8 * i:8 * i + 8], k[:, i:i + 1], v[:, i:i + 1]) for i in range(h)], 1)
    rep = qh // h
    s = torch.einsum("qhd,khd->hqk", q.double(), k.double().repeat_interleave(rep, 1)) / math.sqrt(d)
    s.masked_fill_(torch.ones(n, n, dtype=torch.bool, device=dev).triu(1), -math.inf)
    ref = torch.einsum("hqk,khd->qhd", torch.softmax(s, -1), v.double().repeat_interleave(rep, 1))
    err = [float((x.double() - ref).norm() / ref.norm()) for x in (pairs, single)]
    assert err[0] <= 1.002 * err[1]
