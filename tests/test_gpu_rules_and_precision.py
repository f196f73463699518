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


@pytest.mark.parametrize("d,kb,vb,qh", [(128, 3, 2, 32), (128, 4, 4, 16), (256, 3, 2, 16)])
def test_decode_weighs_the_largest_score_exactly(d, kb, vb, qh, dev):
    """Two tokens that score alike, in records that one warp takes one after the other, and nothing else of weight: the
    softmax reference is the larger score, whose probability is 1 and exact in fp16, and the smaller one was 1 when it came.
    What is left is the ratio of the two: 1.7 units of log2 by queries rounded to fp16 (2^-12 / sqrt(3 d) rms, four sigmas:
    6e-5), and scores of 86 in fp32 (ulp 7.6e-6, a few roundings each: 3e-5), together some 1e-4, where half an ulp of an
    fp16 probability (2.4e-4) comes to 8e-4 of the difference of two values."""
    from turboquant_b200 import _engine as E
    h, nseq, n = 4, 96, 2000
    c = E.LayerConstants(d, kb, vb, dev, seed=5)
    g = torch.Generator().manual_seed(d + kb)
    u = torch.randn(h, d, generator=g)
    u = u / u.norm(dim=-1, keepdim=True)
    k = 0.01 * torch.randn(n, h, d, generator=g)
    a, b = 5, 5 + 16 * 16
    k[a] = k[b] = 8.0 * u
    v = torch.randn(n, h, d, generator=g)
    q = (u.repeat_interleave(qh // h, 0) * 10.0 * math.sqrt(d)).expand(nseq, qh, d).contiguous()
    q = q * (1 + 0.1 * torch.rand(nseq, qh, 1, generator=g))
    k, v, q = k.bfloat16().to(dev), v.bfloat16().to(dev), q.to(dev)
    pool, bt = E.BlockPool(c, h, E.blocks_for(n)), E.identity_block_table(E.blocks_for(n), dev)
    E.store(c, pool, k, v, stride_token=h * d, stride_head=d, n_tokens=n, n_heads=h, block_table=bt, start_pos=0)
    ps = E.pool_to_planes(c, pool, bt, n)
    up = 1 + torch.rand(h, generator=g).to(dev) / 70                # the same vector, up to 1.7 more in log2
    ps.norms[:, b], ps.residual_norms[:, b] = ps.norms[:, a] * up, ps.residual_norms[:, a] * up
    E.planes_to_pool(c, ps, n, pool, bt)
    k64 = _keys64(c, ps.mse_indices, ps.qjl_signs, ps.norms, ps.residual_norms)
    v64 = _unpack(ps.v_data, vb).double().reshape(h, n, -1, 32) * ps.v_scales.double()[..., None] + ps.v_zeros.double()[..., None]
    s = torch.einsum("bhgd,hnd->bhgn", q.double().reshape(nseq, h, -1, d), k64) / math.sqrt(d)
    ref = torch.einsum("bhgn,hnd->bhgd", torch.softmax(s, -1), v64.flatten(-2)).reshape(nseq, qh, d)
    ws = E.Workspace(dev)
    lens = torch.full((nseq,), n, dtype=torch.int32, device=dev)
    out = E.decode(c, pool, ws, q, bt[None].expand(nseq, -1).contiguous(), lens, n, num_splits=1)
    assert ws.status() == 0
    assert float(((out.double() - ref).norm(dim=-1) / ref.norm(dim=-1)).max()) <= 1.5e-4


@pytest.mark.parametrize("d,kb,vb,qh", [(128, 3, 2, 16), (128, 3, 2, 32), (128, 4, 4, 16), (256, 3, 2, 16), (256, 4, 4, 8)])
@pytest.mark.parametrize("records", [1, 56, 57, 73, 124, 125])
def test_decode_on_both_sides_of_the_lines_for_pairs(d, kb, vb, qh, records, dev):
    """Launches of several waves: records one by one and in pairs (also an odd number a warp), a ragged last record, scores
    that climb along the sequence, stale bytes behind the last token."""
    from turboquant_b200 import _engine as E
    h, nseq, n = 4, 50, 16 * records - 3
    c = E.LayerConstants(d, kb, vb, dev, seed=5)
    g = torch.Generator().manual_seed(d + qh + records)
    lens = torch.randint(min(n, 17), n + 1, (nseq,), generator=g)
    lens[0] = n
    q = torch.randn(nseq, qh, d, generator=g).bfloat16().to(dev)
    k = torch.randn(n, h, d, generator=g) + torch.linspace(0, 6, n)[:, None, None] * q[0, :h].float().cpu()[None] / 4
    k, v = k.bfloat16().to(dev), torch.randn(n, h, d, generator=g).bfloat16().to(dev)
    pool = E.BlockPool(c, h, records)
    pool.data.fill_(0x7c)                            # fp16 Inf / NaN patterns
    bt = E.identity_block_table(records, dev)
    E.store(c, pool, k, v, stride_token=h * d, stride_head=d, n_tokens=n, n_heads=h, block_table=bt, start_pos=0)
    table, ws = bt[None].expand(nseq, -1).contiguous(), E.Workspace(dev)
    a, b = (E.decode(c, pool, ws, q, table, lens.int().to(dev), n, num_splits=1, min_history=1, kernel=kern).float() for kern in (0, 1))
    assert ws.status() == 0 and torch.isfinite(a).all()
    assert _cos(a, b) >= 0.99995
    torch.testing.assert_close(a, b, rtol=3e-2, atol=3e-3)


@pytest.mark.parametrize("kb,vb,h,qh", [(3, 2, 8, 32), (4, 2, 2, 8), (3, 4, 8, 64)])
@pytest.mark.parametrize("ring", [0, 32, 33, 128])
@pytest.mark.parametrize("n", [300, 13000])
def test_decode_of_one_sequence_on_both_sides_of_the_lines_for_warps(kb, vb, h, qh, ring, n, dev):
    """Twelve or sixteen warps an SM at head_dim 128 by the ring's length and the records a CTA takes."""
    from turboquant_b200 import _engine as E
    d = 128
    c = E.LayerConstants(d, kb, vb, dev, seed=5)
    k, v = (t.to(dev) for t in O.synth_kv(n + ring, h, d, seed=ring + n, dtype=torch.bfloat16))
    pool, bt = E.BlockPool(c, h, E.blocks_for(n)), E.identity_block_table(E.blocks_for(n), dev)
    E.store(c, pool, k, v, stride_token=h * d, stride_head=d, n_tokens=n, n_heads=h, block_table=bt, start_pos=0)
    q = O.synth_query(1, qh, d, seed=3, dtype=torch.bfloat16).to(dev)
    count = lambda x: torch.tensor([x], dtype=torch.int32, device=dev)  # noqa: E731
    kw = dict(ring_k=k[n:], ring_v=v[n:], ring_lens=count(ring), max_ring_len=ring, ring_stride_token=h * d) if ring else {}
    ws = E.Workspace(dev)
    a, b = (E.decode(c, pool, ws, q, bt[None], count(n), n, kernel=kern, **kw).float() for kern in (0, 1))
    assert ws.status() == 0
    assert _cos(a, b) >= 0.99995
    torch.testing.assert_close(a, b, rtol=3e-2, atol=3e-3)


def test_planes_of_another_size_type_or_place_are_not_read(dev):
    """What the kernels on plain rows would read out of range goes the general way, which raises or moves it."""
    from turboquant_b200 import TurboQuantProd
    from turboquant_b200.kv_cache import dequantize_values, quantize_values
    z3, z4 = TurboQuantProd(128, 3, device=dev), TurboQuantProd(128, 4, device=dev)
    x = torch.randn(2, 50, 128, device=dev)
    kq, q = z3.quantize(x), torch.randn(2, 3, 128, device=dev)
    for bad in (kq._replace(qjl_signs=kq.qjl_signs[:, :20].contiguous()), kq._replace(norms=kq.norms[:1]),
                kq._replace(residual_norms=kq.residual_norms[:, ::2].contiguous())):
        for call in (lambda: z3.dequantize(bad), lambda: z3.attention_score(q, bad)):
            with pytest.raises(RuntimeError):
                call()
    with pytest.raises(RuntimeError):                  # 3-bit codes in a 4-bit quantiser
        z4.dequantize(kq)
    there = kq._replace(norms=kq.norms.cpu(), residual_norms=kq.residual_norms.cpu())
    assert torch.equal(z3.dequantize(there), z3.dequantize(kq)) or \
        torch.allclose(z3.dequantize(there), z3.dequantize(kq), rtol=1e-4, atol=1e-4)
    wide = kq._replace(mse_indices=kq.mse_indices.int())
    assert torch.allclose(z3.dequantize(wide), z3.dequantize(kq), rtol=1e-4, atol=1e-4)
    vq = quantize_values(x, 2)
    with pytest.raises(RuntimeError):
        dequantize_values(vq._replace(scales=vq.scales[:, :20].contiguous()))
    assert torch.equal(dequantize_values(vq._replace(zeros=vq.zeros.half())), dequantize_values(vq))


@pytest.mark.parametrize("n_q", [128, 129])
def test_cache_object_with_many_queries(n_q, dev):
    """Both sides of the line between the attend kernel and the matrix product on dequantised values; no scratch for a call
    that is declined, the logits' scratch is the prepared queries."""
    from turboquant_b200 import TurboQuantKVCache, _engine as E
    d, h, n = 128, 3, 700
    cache = TurboQuantKVCache(d, 3, 2, buffer_size=32, device=dev, dtype=torch.float32)
    g = torch.Generator().manual_seed(n_q)
    k, v = (torch.randn(1, h, n, d, generator=g).to(dev) for _ in range(2))
    cache.prefill(k, v)
    q, w = torch.randn(1, h, n_q, d, generator=g).to(dev), torch.softmax(torch.randn(1, h, n_q, n, generator=g), -1).to(dev)
    m = cache._n_quant
    logits = cache.attention_scores(q)
    scratch = cache._ws_attn.buf.numel()
    assert scratch <= 32768 + h * n_q * 2 * d * 4
    out = cache.attend(w)
    assert (cache._ws_attn.buf.numel() == scratch) == (n_q > 128)
    keys = torch.cat((E.dequant_keys(cache.consts, cache._pool, cache._bt, m).reshape(1, h, m, d), k[..., m:, :]), -2).double()
    vals = torch.cat((E.dequant_values(cache.consts, cache._pool, cache._bt, m).reshape(1, h, m, d), v[..., m:, :]), -2).double()
    for got, ref in ((logits, q.double() @ keys.transpose(-1, -2) / math.sqrt(d)), (out, w.double() @ vals)):
        assert float((got.double() - ref).norm() / ref.norm()) <= 2e-6      # fp32 sums of some hundred terms


@pytest.mark.parametrize("kb,vb", [(4, 2), (3, 4)])
def test_d256_wide_records_are_as_exact_as_the_fp32_store(kb, vb, dev):
    """Codes next to a boundary and sign bits next to zero that come out otherwise than in 64 bits: not more than from the
    fp32 kernel, up to three standard deviations of the two counts (bf16 limbs gave six to twelve times as many)."""
    from turboquant_b200 import _engine as E
    n, h, d = 16384, 8, 256
    g = torch.Generator(device=dev)
    g.manual_seed(11)
    x = (torch.randn(n, h, d, generator=g, device=dev) * torch.exp(0.5 * torch.randn(d, generator=g, device=dev))).bfloat16()
    wrong = []
    for tensor_cores in (True, False):
        c = E.LayerConstants(d, kb, vb, dev, tensor_core_store=tensor_cores)
        pool, bt = E.BlockPool(c, h, E.blocks_for(n)), E.identity_block_table(E.blocks_for(n), dev)
        E.store(c, pool, x, x, stride_token=h * d, stride_head=d, n_tokens=n, n_heads=h, block_table=bt)
        ps = E.pool_to_planes(c, pool, bt, n)
        wrong.append([sum(w) for w in zip(*(_wrong(c, x[:, i], ps.mse_indices[i], ps.qjl_signs[i]) for i in range(h)))])
    for fast, exact in zip(*wrong):
        assert fast <= exact + 3 * math.sqrt(fast + exact), wrong
    assert E.store_status() == 0


def test_d256_wide_store_without_fp16_operands(dev):
    """A rotation whose residuals would leave fp16's range has no operands for the tensor-core kernel: the fp32 one runs."""
    from turboquant_b200 import _engine as E
    n, h, d = 100, 2, 256
    x = torch.randn(n, h, d, generator=torch.Generator().manual_seed(1)).bfloat16().to(dev)
    pi = 20.0 * E.LayerConstants(d, 4, 2, dev).Pi
    planes = []
    for tensor_cores in (True, False):
        c = E.LayerConstants(d, 4, 2, dev, Pi=pi, tensor_core_store=tensor_cores)
        assert c.rows_limbs is None
        pool, bt = E.BlockPool(c, h, E.blocks_for(n)), E.identity_block_table(E.blocks_for(n), dev)
        E.store(c, pool, x, x, stride_token=h * d, stride_head=d, n_tokens=n, n_heads=h, block_table=bt)
        planes.append(E.pool_to_planes(c, pool, bt, n))
    for f in ("mse_indices", "qjl_signs", "norms", "residual_norms"):
        assert torch.equal(getattr(planes[0], f), getattr(planes[1], f))


@pytest.mark.parametrize("bits", [3, 4])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_key_rows_kernels_are_as_exact_as_fp32(bits, dtype, dev):
    """Quantising and dequantising plain rows by limb products against 64 bits and against the fp32 kernels on records:
    the same codes, not more wrong sign bits (three standard deviations), no larger error of the rows that come back."""
    from turboquant_b200 import TurboQuantProd, _engine as E
    n = 200000
    z = TurboQuantProd(128, bits, device=dev)
    g = torch.Generator(device=dev)
    g.manual_seed(13)
    x = (torch.randn(n, 128, generator=g, device=dev) * torch.exp(0.5 * torch.randn(128, generator=g, device=dev))).to(dtype)
    kq, ps = z.quantize(x), z._compress_rows(x)[2]
    assert torch.equal(kq.mse_indices, ps.mse_indices[0])
    fast, exact = (_wrong(z.consts, x, s.mse_indices.view(n, -1), s.qjl_signs.view(n, -1))[1] for s in (kq, ps))
    assert fast <= exact + 3 * math.sqrt(fast + exact)
    ref = _keys64(z.consts, kq.mse_indices, kq.qjl_signs, kq.norms, kq.residual_norms)
    pool, bt, _, m = z._pool_from(kq.mse_indices, kq.qjl_signs, kq.norms, kq.residual_norms)
    err = [float((t.reshape(n, 128).double() - ref).norm() / ref.norm()) for t in (z.dequantize(kq), E.dequant_keys(z.consts, pool, bt, m))]
    assert err[0] <= err[1]


@pytest.mark.parametrize("bits", [3, 4])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_key_rows_on_the_decision_boundaries(bits, dtype, dev):
    """Rows with half of their rotated coordinates on a boundary, where the limb product decides otherwise than the fp32
    chain in many a row, which is then redone as a whole: codes, residual norms and sign bits are the fp32 store's."""
    from turboquant_b200 import TurboQuantProd
    n = 3000
    z = TurboQuantProd(128, bits, device=dev)
    g = torch.Generator().manual_seed(bits)
    inner = z.consts.boundaries_cpu[1:-1].double()
    y = inner[torch.randint(0, len(inner), (n, 128), generator=g)]
    rest = torch.randn(n, 64, generator=g).double()
    room = (1 - y[:, :64].pow(2).sum(1, keepdim=True)).clamp_min(1e-3).sqrt()
    y[:, 64:] = rest / rest.norm(dim=1, keepdim=True) * room
    x = (y @ z.consts.Pi.cpu().double()).to(dtype).to(dev)
    kq, ps = z.quantize(x), z._compress_rows(x)[2]
    assert torch.equal(kq.mse_indices, ps.mse_indices[0])
    assert torch.equal(kq.norms.half(), ps.norms[0])
    torch.testing.assert_close(kq.residual_norms, ps.residual_norms[0].float(), rtol=1.1e-3, atol=0)   # an ulp of fp16
    assert _bit_frac(kq.qjl_signs, ps.qjl_signs[0]) <= 2e-5     # sums of 128 terms within 1e-6 of zero


def test_captured_decode_reads_its_lengths_at_replay(dev):
    """A step captured at the longest history and replayed after a shorter one took its place attends to the shorter one;
    a captured fused step appends behind the tokens that the ring then holds."""
    from turboquant_b200 import CompressedKVStore, KVCaptureEngine, compute_hybrid_attention
    d, h, qh, n = 128, 4, 16, 600
    k, v = (t.to(dev) for t in O.synth_kv(n + 40, h, d, seed=1, dtype=torch.bfloat16))
    q = O.synth_query(1, qh, d, seed=2, dtype=torch.bfloat16).to(dev)
    store = CompressedKVStore(d, h, 3, 2, device=dev, capacity_tokens=n)
    engine = KVCaptureEngine(store, ring_capacity=64, device=dev)
    store.append_chunk(k[:n], v[:n])
    engine.ingest_decode(k[n:n + 20], v[n:n + 20], 20)
    rk, rv = engine.ring.peek()
    store.seq_len_device, engine.ring.device_len()
    compute_hybrid_attention(q, store, rk, rv, qh)      # scratch at its size
    one, step = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(one):
        out = compute_hybrid_attention(q, store, rk, rv, qh)
    store.reset()
    store.append_chunk(k[:200], v[:200])
    store.seq_len_device
    one.replay()
    torch.cuda.synchronize()
    want = compute_hybrid_attention(q, store, rk, rv, qh)
    torch.testing.assert_close(out.float(), want.float(), rtol=2e-2, atol=2e-3)

    engine.decode_step(q, k[n + 20:n + 21], v[n + 20:n + 21], qh)
    engine.ring.device_len()
    with torch.cuda.graph(step):
        engine.decode_step(q, k[n + 21:n + 22], v[n + 21:n + 22], qh)
    step.replay()
    step.replay()                                       # the second behind the first
    torch.cuda.synchronize()
    keys = engine.ring.storage[0]
    assert torch.equal(keys[21], k[n + 21]) and torch.equal(keys[22], k[n + 21])


def test_cache_object_takes_weights_that_broadcast(dev):
    """Weights shared by the heads or the batch, or without a batch: what the matrix products broadcast or refuse."""
    from turboquant_b200 import TurboQuantKVCache
    g = torch.Generator().manual_seed(4)
    for b, shapes, bad in ((2, ((2, 3, 2), (2, 1, 2), (1, 3, 2), (1, 1, 2)), ((3, 2, 2), (6, 2))), (1, ((1, 3, 2), (3, 2), (3, 1, 2)), ((1, 2, 2), (2, 2)))):
        cache = TurboQuantKVCache(128, 3, 2, buffer_size=16, device=dev, dtype=torch.float32)
        k, v = (torch.randn(b, 3, 200, 128, generator=g).to(dev) for _ in range(2))
        cache.prefill(k, v)
        eye = torch.eye(200, device=dev).expand(b, 3, 200, 200).contiguous()
        values = torch.cat([cache.attend(eye[..., i:i + 100, :].contiguous()) for i in (0, 100)], -2)
        for lead in shapes:
            w = torch.softmax(torch.randn(*lead, 200, generator=g), -1).to(dev)
            got = cache.attend(w)
            want = torch.matmul(w, values)
            assert got.shape == want.shape
            torch.testing.assert_close(got, want, rtol=1e-4, atol=1e-5)
        for lead in bad:
            with pytest.raises(RuntimeError):
                cache.attend(torch.ones(*lead, 200, device=dev))


def test_hybrid_attention_on_strided_tensors_equals_contiguous_ones(dev):
    from turboquant_b200 import CompressedKVStore, compute_hybrid_attention
    g = torch.Generator(device=dev)
    g.manual_seed(8)
    wide = lambda *s: torch.randn(*s, 256, generator=g, device=dev).bfloat16()[..., :128]  # noqa: E731
    store = CompressedKVStore(128, 4, 3, 2, device=dev, capacity_tokens=500)
    store.append_chunk(wide(500, 4).contiguous(), wide(500, 4).contiguous())
    q, rk, rv = wide(3, 16), wide(30, 4), wide(30, 4)
    want = compute_hybrid_attention(q.contiguous(), store, rk.contiguous(), rv.contiguous(), 16)
    assert torch.equal(compute_hybrid_attention(q, store, rk, rv, 16), want)
    assert torch.equal(compute_hybrid_attention(q, store, rk.contiguous(), rv, 16), want)


def test_a_host_tensor_is_no_place_for_a_result(dev):
    from turboquant_b200 import CompressedCacheSpec, CompressedPagedKVCache
    cache = CompressedPagedKVCache.allocate(CompressedCacheSpec(128, 2, 3, 2), 4, dev)
    k = torch.randn(40, 2, 128, device=dev).bfloat16()
    cache.write(k, k, torch.arange(40, device=dev))
    q, table, lens = torch.randn(1, 8, 128, device=dev).bfloat16(), torch.arange(4, dtype=torch.int32, device=dev)[None], \
        torch.tensor([40], dtype=torch.int32, device=dev)
    with pytest.raises((TypeError, ValueError, RuntimeError)):
        cache.decode(q, table, lens, 40, out=torch.empty(1, 8, 128, dtype=torch.bfloat16))
    out = torch.empty_like(q)
    assert cache.decode(q, table, lens, 40, out=out) is out


@pytest.mark.parametrize("kb,vb,qh", [(3, 2, 32), (3, 2, 64), (4, 4, 32)])
def test_host_step_and_device_step_give_the_same_bits(kb, vb, qh, dev):
    """One sequence at head_dim 128 from 33 ring tokens on: the same number of warps, so the same softmax references and the
    same rounding of every probability, wherever the query lies.  (With twelve warps in the place of sixteen the outputs
    differ by 5e-4 and the error against 64 bits is 2 % larger.)"""
    from turboquant_b200 import CompressedKVStore, KVCaptureEngine
    h, d, n = 8, 128, 4096
    g = torch.Generator(device=dev).manual_seed(kb + qh)
    k, v = (torch.randn(n + 128, h, d, generator=g, device=dev, dtype=torch.bfloat16) for _ in range(2))
    q = torch.randn(1, qh, d, generator=g, device=dev, dtype=torch.bfloat16)
    engines = []
    for _ in range(2):
        e = KVCaptureEngine(CompressedKVStore(d, h, kb, vb, device=dev, capacity_tokens=n), ring_capacity=128, device=dev)
        e.store.append_chunk(k[:n], v[:n])
        e.ring.write(k[n:n + 32], v[n:n + 32], 32)
        engines.append(e)
    host_out = torch.zeros(qh * d, dtype=torch.bfloat16).pin_memory()
    for i in range(n + 32, n + 128):
        out = engines[0].decode_step(q, k[i:i + 1], v[i:i + 1], qh)
        rows = torch.cat([t.reshape(-1) for t in (k[i], v[i], q)]).cpu().pin_memory()
        engines[1].decode_step_host(rows, host_out, qh)
        torch.cuda.synchronize()
        assert torch.equal(out.flatten().cpu(), host_out), engines[0].ring.size
