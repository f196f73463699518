"""Edges of the kernels' splits - ring tokens over warps, partial results over threads, queries over CTAs, rows over tiles -
against 64-bit arithmetic on what the records hold."""

import math

import pytest
import torch

from tests.test_gpu_rules_and_precision import _keys64, _unpack

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    return torch.device("cuda:0")


def _history64(consts, planes, n, vb):
    """Dequantised keys and values (H, n, D) in 64 bits."""
    k = _keys64(consts, planes.mse_indices[:, :n], planes.qjl_signs[:, :n], planes.norms[:, :n], planes.residual_norms[:, :n])
    code = _unpack(planes.v_data[:, :n], vb).double()
    scale, zero = (t[:, :n].double().repeat_interleave(32, -1) for t in (planes.v_scales, planes.v_zeros))
    return k, code * scale + zero


def _attend64(q, k, v, group):
    """q (T, Qh, D), k / v (H, N, D) -> (T, Qh, D)"""
    k, v = (t.repeat_interleave(group, 0) for t in (k, v))
    p = torch.softmax(torch.einsum("thd,hnd->thn", q.double(), k) / math.sqrt(q.shape[-1]), -1)
    return torch.einsum("thn,hnd->thd", p, v)


def _rel(got, want):
    return float((got.double() - want).norm() / want.norm())


@pytest.mark.parametrize("d,h,qh", [(128, 8, 32), (128, 2, 16), (128, 3, 3), (256, 4, 16), (256, 2, 16)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_ring_lengths_on_both_sides_of_every_split(d, h, qh, dtype, dev):
    """Ring tokens alone (a history below 16 tokens does not count): fp32 all the way.  A score is a sum of D products,
    wrong by at most (log2(D) + 8) 2^-24 sum |q k| / sqrt(D) <= 16 * 6e-8 * 13 = 1.2e-5, which is the relative error of a
    probability; the 2^-22 of the exponential's approximation and the output's own rounding come on top."""
    from turboquant_b200 import CompressedKVStore, compute_hybrid_attention
    store = CompressedKVStore(d, h, 3, 2, device=dev)
    g = torch.Generator(device=dev).manual_seed(d + qh)
    r_max = 256
    k, v = (torch.randn(r_max, h, d, generator=g, device=dev, dtype=dtype) for _ in range(2))
    q = torch.randn(1, qh, d, generator=g, device=dev, dtype=dtype)
    tol = 3e-5 + {torch.float32: 0.0, torch.bfloat16: 2.0 ** -9, torch.float16: 2.0 ** -12}[dtype]
    for r in (1, 2, 3, 23, 24, 25, 31, 32, 33, 47, 48, 49, 63, 64, 65, 95, 97, 127, 128, 129, 191, 193, 256):
        out = compute_hybrid_attention(q, store, k[:r], v[:r], qh)
        want = _attend64(q, k[:r].double().transpose(0, 1), v[:r].double().transpose(0, 1), qh // h)
        assert _rel(out, want) <= tol, r
    assert store.workspace.status() == 0


@pytest.mark.parametrize("d,h,qh,kb,vb", [(128, 2, 8, 3, 2), (128, 1, 8, 4, 4), (256, 1, 4, 3, 2), (256, 2, 16, 4, 2)])
def test_merge_of_any_number_of_partial_results(d, h, qh, kb, vb, dev):
    """One CTA up to more slots than a warp looks at twice, with and without ring slots between.  Probabilities are fp16
    (2^-12 each, 5e-4 measured for whole outputs), so twice what they give bounds a slot left out or taken twice, which
    would cost at least 1 / 140."""
    from turboquant_b200 import CompressedKVStore, _engine as E
    n = 2240
    store = CompressedKVStore(d, h, kb, vb, device=dev, capacity_tokens=n)
    g = torch.Generator(device=dev).manual_seed(7 * d + qh)
    k, v = (torch.randn(n, h, d, generator=g, device=dev, dtype=torch.bfloat16) for _ in range(2))
    store.append_chunk(k, v)
    rk, rv = (torch.randn(70, h, d, generator=g, device=dev, dtype=torch.bfloat16) for _ in range(2))
    q = torch.randn(1, qh, d, generator=g, device=dev)
    k64, v64 = _history64(store.consts, E.pool_to_planes(store.consts, store.pool, store.block_table, n), n, vb)
    lens, ring_lens = (torch.tensor([x], dtype=torch.int32, device=dev) for x in (n, 70))
    for splits in (1, 2, 3, 4, 13, 14, 37, 40, 63, 64, 65, 100, 128, 140):
        for ring in (False, True):
            kw = dict(ring_k=rk, ring_v=rv, ring_lens=ring_lens, max_ring_len=70, ring_stride_token=h * d) if ring else {}
            out = E.decode(store.consts, store.pool, store.workspace, q, store.block_table[None], lens, n, num_splits=splits, **kw)
            ks, vs = ((torch.cat((a, b.double().transpose(0, 1)), 1) if ring else a) for a, b in ((k64, rk), (v64, rv)))
            assert _rel(out, _attend64(q, ks, vs, qh // h)) <= 1e-3, (splits, ring)
    assert store.workspace.status() == 0


@pytest.mark.parametrize("d,kb,vb", [(128, 3, 2), (128, 4, 4), (256, 3, 4), (256, 4, 2)])
@pytest.mark.parametrize("n,buf", [(1, 1), (63, 0), (65, 5), (129, 64), (1000, 129)])
def test_cache_object_for_every_group_of_queries(d, kb, vb, n, buf, dev):
    """Sums of up to 1129 fp32 products: (log2(1129) + 8) 2^-24 = 1.1e-6 of the sum of magnitudes, which for random signs is
    some sqrt(1129) times the sum."""
    from turboquant_b200 import TurboQuantKVCache, _engine as E
    g = torch.Generator(device=dev).manual_seed(n + d)
    cache = TurboQuantKVCache(d, kb, vb, buffer_size=max(buf, 1), device=dev, dtype=torch.float16)
    k, v = (torch.randn(1, 2, n + buf, d, generator=g, device=dev, dtype=torch.float16) for _ in range(2))
    if buf:
        cache.prefill(k, v)
    else:
        cache._append_compressed(k, v)
    k64, v64 = _history64(cache.consts, E.pool_to_planes(cache.consts, cache._pool, cache._bt, n), n, vb)
    k64, v64 = (torch.cat((a, b[0, :, n:].double()), 1) for a, b in ((k64, k), (v64, v)))
    for n_q in (1, 2, 3, 4, 5, 8, 9):
        q = torch.randn(1, 2, n_q, d, generator=g, device=dev, dtype=torch.float16)
        logits = cache.attention_scores(q)
        want = torch.einsum("hqd,hnd->hqn", q[0].double(), k64) / math.sqrt(d)
        assert logits.dtype == torch.float32 and _rel(logits[0], want) <= 2e-6, n_q
        w = torch.softmax(logits, -1)
        assert _rel(cache.attend(w)[0], torch.einsum("hqn,hnd->hqd", w[0].double(), v64)) <= 4e-6, n_q


@pytest.mark.parametrize("bits", [3, 4])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_key_rows_do_not_depend_on_their_place(bits, dtype, dev):
    """The rows of one call are the rows of another: ends of row groups, tiles and waves."""
    from turboquant_b200 import TurboQuantProd
    z = TurboQuantProd(128, bits, device=dev)
    n_all = 148 * 128 + 300
    x = torch.randn(n_all, 128, generator=torch.Generator(device=dev).manual_seed(bits), device=dev).to(dtype)
    x[5] = 0
    full = z.quantize(x)
    back = z.dequantize(full)
    for lo, n in ((0, 1), (3, 7), (0, 8), (1, 9), (2, 15), (0, 16), (0, 17), (100, 127), (0, 128), (7, 129), (0, 255), (11, 148 * 128), (0, 148 * 128 + 1)):
        part = z.quantize(x[lo:lo + n])
        for a, b in zip(part[:4], full[:4]):
            assert torch.equal(a, b[lo:lo + n]), (lo, n)
        assert torch.equal(z.dequantize(part), back[lo:lo + n]), (lo, n)


@pytest.mark.parametrize("d,bits", [(128, 2), (128, 4), (256, 2), (256, 4)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_value_rows_for_any_number_of_groups(d, bits, dtype, dev):
    """Codes, scales and zero points of n rows against the same arithmetic in torch, exactly; values back to the rounding of
    one multiply-add."""
    from turboquant_b200.kv_cache import dequantize_values, quantize_values
    g = torch.Generator(device=dev).manual_seed(d + bits)
    for n in (1, 2, 15, 16, 17, 63, 65, 1000):
        v = torch.randn(1, n, d, generator=g, device=dev).to(dtype)
        v[0, 0, :32] = 1.5                       # a group without a range
        out = quantize_values(v, bits=bits)
        x = v.view(n, d // 32, 32)
        lo, hi = x.amin(-1, keepdim=True), x.amax(-1, keepdim=True)
        scale = ((hi - lo) / torch.full_like(hi, 2 ** bits - 1)).clamp(min=1e-10)   # by a tensor: a number is multiplied by its inverse
        code = ((x - lo) / scale).round().clamp(0, 2 ** bits - 1).nan_to_num(0).long().view(n, d)   # 0 / 0 where fp16 has no 1e-10
        assert torch.equal(_unpack(out.data.view(n, -1), bits), code)
        assert torch.equal(out.scales.view(n, -1), scale[..., 0].half().to(dtype)) and torch.equal(out.zeros.view(n, -1), lo[..., 0].half().to(dtype))
        s64, z64 = (t.view(n, -1).half().double().repeat_interleave(32, -1) for t in (out.scales, out.zeros))
        want = code.double() * s64 + z64
        assert float((dequantize_values(out).view(n, d).double() - want).abs().max()) <= 2.0 ** -22 * float(want.abs().max() + s64.max() * (2 ** bits))


@pytest.mark.parametrize("kb,vb", [(4, 2), (3, 4), (4, 4)])
@pytest.mark.parametrize("n", [1, 127, 129, 700])
def test_d256_wide_records_from_a_paged_cache(kb, vb, n, dev):
    """The table-walking launch writes what the launch on gathered rows writes; without `any_width` it is refused as before."""
    from turboquant_b200 import CompressedKVStore, _engine as E
    h, bs, d = 3, 16, 256
    g = torch.Generator(device=dev).manual_seed(n)
    used = (n + bs - 1) // bs
    table = torch.randperm(used + 5, generator=g, device=dev)[:used].int()
    cache = torch.randn(2, used + 5, bs, h, d, generator=g, device=dev, dtype=torch.bfloat16)
    k, v = (cache[i][table.long()].flatten(0, 1)[:n] for i in range(2))
    a = CompressedKVStore(d, h, kb, vb, device=dev, capacity_tokens=n)
    a.append_chunk(k, v)
    pool = E.BlockPool(a.consts, h, E.blocks_for(n))
    args = dict(src_block_table=table, n_tokens=n, block_table=E.identity_block_table(E.blocks_for(n), dev))
    assert not E.store_paged(a.consts, pool, cache[0], cache[1], **args)
    assert E.store_paged(a.consts, pool, cache[0], cache[1], any_width=True, **args)
    size = E.blocks_for(n) * h * a.consts.block_bytes
    assert torch.equal(pool.data[:size], a.pool.data[:size]) and E.store_status() == 0


@pytest.mark.parametrize("bs", [1, 5, 16, 48])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_ring_is_filled_from_a_paged_cache(bs, dtype, dev):
    """The last tokens of a prompt, into an empty ring and behind tokens that it holds; a full ring or a table of another type
    takes the general way with the same result."""
    from turboquant_b200 import CompressedKVStore, KVCaptureEngine
    h, d, cap = 2, 128, 32
    g = torch.Generator(device=dev).manual_seed(bs)
    for n, held, wide in ((1, 0, False), (31, 0, False), (32, 0, True), (20, 12, False), (20, 13, False), (75, 0, False), (75, 3, False)):
        used = (n + bs - 1) // bs
        table = torch.randperm(used + 3, generator=g, device=dev)[:used].to(torch.int64 if wide else torch.int32)
        cache = torch.randn(2, used + 3, bs, h, d, generator=g, device=dev).to(dtype)
        k, v = (cache[i][table.long()].flatten(0, 1)[:n] for i in range(2))
        k0, v0 = (torch.randn(max(held, 1), h, d, generator=g, device=dev).to(dtype) for _ in range(2))
        both = []
        for paged in (True, False):
            e = KVCaptureEngine(CompressedKVStore(d, h, 3, 2, device=dev), ring_capacity=cap, device=dev, dtype=dtype)
            if held:
                e.ring.write(k0[:held], v0[:held], held)
            if paged:
                e.ingest_prefill_from_paged_cache(cache, n, table, bs)
            else:
                m = max(n - cap, 0)
                if m:
                    e.store.append_chunk(k[:m], v[:m])
                e.ring.write(k[m:], v[m:], n - m)
            both.append(e)
        a, b = both
        assert (a.ring.size, a.ring.total_written, a.store.num_tokens) == (b.ring.size, b.ring.total_written, b.store.num_tokens)
        assert all(torch.equal(x, y) for x, y in zip(a.ring.peek(), b.ring.peek())), (n, held)


@pytest.mark.parametrize("d,bits", [(128, 3), (128, 4), (256, 3), (256, 4)])
@pytest.mark.parametrize("mid", [0.0, 1e-25, -2e-25, 9e-26, -1e-30, 1e-39])
def test_store_with_a_middle_boundary_next_to_zero(d, bits, mid, dev):
    """The tensor-core kernels scale differences up and flush what is below the normal numbers, so a code book whose middle
    boundary lies between 0 and 1e-25 is the fp32 kernel's, byte for byte.  With others at most 1e-4 of the codes and of the
    sign bits differ, as with any code book: a byte holds up to four codes, or eight bits."""
    from turboquant_b200 import _engine as E
    n, h = 300, 2
    base = E.LayerConstants(d, bits, 2, dev)
    edges = base.boundaries_cpu.clone()
    edges[len(edges) // 2] = mid
    g = torch.Generator(device=dev).manual_seed(d + bits)
    k, v = (torch.randn(n, h, d, generator=g, device=dev, dtype=torch.bfloat16) for _ in range(2))
    pools = []
    for fast in (True, False):
        c = E.LayerConstants(d, bits, 2, dev, centroids=base.centroids_cpu, boundaries=edges, tensor_core_store=fast)
        pool = E.BlockPool(c, h, E.blocks_for(n))
        E.store(c, pool, k, v, stride_token=h * d, stride_head=d, n_tokens=n, n_heads=h,
                block_table=E.identity_block_table(E.blocks_for(n), dev))
        pools.append((pool.data[:E.blocks_for(n) * h * c.block_bytes].clone(),
                      E.pool_to_planes(c, pool, E.identity_block_table(E.blocks_for(n), dev), n)))
    (a, pa), (b, pb) = pools
    if 0 < abs(mid) < 1e-25:
        assert torch.equal(a, b)
    assert float((pa.mse_indices[:, :n] != pb.mse_indices[:, :n]).float().mean()) <= 4e-4
    assert float((pa.qjl_signs[:, :n] != pb.qjl_signs[:, :n]).float().mean()) <= 8e-4


@pytest.mark.parametrize("d,kb,vb", [(128, 3, 2), (128, 4, 4), (256, 3, 2), (256, 4, 2)])
def test_store_right_behind_the_call_that_writes_its_last_row(d, kb, vb, dev):
    """The decode call writes a token into the ring and the store behind it, which begins under it, reads that row."""
    from turboquant_b200 import CompressedKVStore, KVCaptureEngine
    h, cap, n = 2, 48, 4000
    g = torch.Generator(device=dev).manual_seed(d + kb)
    k, v = (torch.randn(n + cap, h, d, generator=g, device=dev, dtype=torch.bfloat16) for _ in range(2))
    q = torch.randn(1, 4 * h, d, generator=g, device=dev, dtype=torch.bfloat16)
    want = CompressedKVStore(d, h, kb, vb, device=dev, capacity_tokens=n + cap)
    for lo, hi in ((0, n), (n, n + cap)):
        want.append_chunk(k[lo:hi], v[lo:hi])
    size = (n + cap) // 16 * h * want.consts.block_bytes
    for _ in range(10):
        engine = KVCaptureEngine(CompressedKVStore(d, h, kb, vb, device=dev, capacity_tokens=n + cap), ring_capacity=cap, device=dev)
        engine.store.append_chunk(k[:n], v[:n])
        engine.ingest_decode(k[n:-1], v[n:-1], cap - 1)
        engine.decode_step(q, k[-1:], v[-1:], 4 * h)
        engine.flush()
        assert torch.equal(engine.store.pool.data[:size], want.pool.data[:size])


def _others_launch(dev, streams):
    """Something of the library on each of the streams."""
    from turboquant_b200.kv_cache import quantize_values
    v = torch.randn(1, 4, 128, device=dev, dtype=torch.bfloat16)
    for s in streams:
        with torch.cuda.stream(s):
            quantize_values(v, bits=2)


@pytest.mark.parametrize("d,kb,vb", [(128, 3, 2), (256, 4, 4)])
def test_scores_right_behind_a_store_with_nine_streams_between(d, kb, vb, dev):
    """A store lets what follows on its stream begin at once.  With queued work in front of it and launches on more streams than
    are kept in mind behind it, neither the cache object nor the decode may read records that are not written."""
    from turboquant_b200 import CompressedKVStore, TurboQuantKVCache, compute_hybrid_attention
    n, h = 3000, 4
    g = torch.Generator(device=dev).manual_seed(d + kb)
    k, v = (torch.randn(1, h, n, d, generator=g, device=dev, dtype=torch.bfloat16) for _ in range(2))
    q = torch.randn(1, h, 1, d, generator=g, device=dev, dtype=torch.bfloat16)
    qd = torch.randn(1, 4 * h, d, generator=g, device=dev, dtype=torch.bfloat16)
    rows_k, rows_v = (t[0].transpose(0, 1) for t in (k, v))
    mine, *others = (torch.cuda.Stream(dev) for _ in range(10))
    _others_launch(dev, others)
    torch.cuda.synchronize()
    for _ in range(8):
        cache = TurboQuantKVCache(d, kb, vb, buffer_size=8, device=dev, dtype=torch.bfloat16)
        store = CompressedKVStore(d, h, kb, vb, device=dev, capacity_tokens=n)
        torch.cuda.synchronize()
        with torch.cuda.stream(mine):
            torch.cuda._sleep(4_000_000)          # about 2 ms, so that everything below is queued behind it
            cache.prefill(k, v)
        _others_launch(dev, others)
        with torch.cuda.stream(mine):
            logits = cache.attention_scores(q)
            torch.cuda._sleep(4_000_000)
            store.append_chunk(rows_k, rows_v)
        _others_launch(dev, others)
        with torch.cuda.stream(mine):
            out = compute_hybrid_attention(qd, store, None, None, 4 * h)
        torch.cuda.synchronize()
        assert torch.equal(logits, cache.attention_scores(q))
        assert torch.equal(out, compute_hybrid_attention(qd, store, None, None, 4 * h))


@pytest.mark.parametrize("d,kb,vb", [(128, 3, 2), (256, 4, 4)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32, torch.bfloat16])
def test_scores_right_behind_a_flush(d, kb, vb, dtype, dev):
    """History, scores and output with nothing launched in between, over a pool that grows on the way, and the same again once
    everything is at rest."""
    from turboquant_b200 import TurboQuantKVCache
    h, n = 2, 2600
    g = torch.Generator(device=dev).manual_seed(d + kb)
    k, v = (torch.randn(1, h, n, d, generator=g, device=dev, dtype=dtype) for _ in range(2))
    q = torch.randn(1, h, 2, d, generator=g, device=dev, dtype=dtype)
    for _ in range(5):
        cache = TurboQuantKVCache(d, kb, vb, buffer_size=4, device=dev, dtype=dtype)
        got = []
        cache.prefill(k[..., :600, :], v[..., :600, :])
        for at in (600, 1100, 1101, 2400):       # 1024 tokens of room, then twice that, then more
            got.append((cache._n_quant, cache.attention_scores(q)))
            m = {600: 500, 1100: 1, 1101: 1299, 2400: 200}[at]
            cache.append(k[..., at:at + m, :], v[..., at:at + m, :])
        last = cache.attention_scores(q)
        torch.cuda.synchronize()
        assert cache._n_quant == n - 4
        full = cache.attention_scores(q)
        assert torch.equal(last, full)
        for m, logits in got:
            assert torch.equal(logits[..., :m], full[..., :m]), m


@pytest.mark.parametrize("bad", [-1, 9, 2 ** 30])
@pytest.mark.parametrize("n", [20, 75])
def test_ring_filled_through_a_table_with_a_bad_index(bad, n, dev):
    """The tokens of that block become zeros - nothing of what the ring held for another sequence - the others arrive, and the
    engine's next calls raise until it is reset."""
    from turboquant_b200 import CompressedKVStore, KVCaptureEngine, _engine as E
    h, d, cap, bs = 2, 128, 32, 16
    g = torch.Generator(device=dev).manual_seed(n)
    cache = torch.randn(2, 9, bs, h, d, generator=g, device=dev, dtype=torch.bfloat16)
    used = (n + bs - 1) // bs
    table = torch.randperm(9, generator=g, device=dev)[:used].int()
    wrong = table.clone()
    wrong[-1] = bad
    e = KVCaptureEngine(CompressedKVStore(d, h, 3, 2, device=dev), ring_capacity=cap, device=dev)
    e.ring.write(*(torch.full((cap, h, d), 7.0, device=dev, dtype=torch.bfloat16) for _ in range(2)), cap)
    for tab in (table, wrong, table):
        e.reset()
        e.ingest_prefill_from_paged_cache(cache, n, tab, bs)
        torch.cuda.synchronize()
        m = min(n, cap)
        want = cache[:, table.long()].flatten(1, 2)[:, n - m:n].clone()
        if tab is wrong:
            want[:, bs * (used - 1) - n:] = 0
            row = torch.zeros(1, h, d, device=dev, dtype=torch.bfloat16)
            q = torch.zeros(1, 4 * h, d, device=dev, dtype=torch.bfloat16)
            for call in (e.ring.peek, e.flush, e.ring.drain, lambda: e.ingest_decode(row, row, 1), lambda: e.ring.write_one(row, row),
                         lambda: e.decode_step(q, row, row, 4 * h)):
                with pytest.raises(IndexError):
                    call()
            assert E.store_status() == -7
        else:
            assert e.ring.peek()[0].shape[0] == m and E.store_status() == 0
        assert torch.equal(e.ring._keys[:m], want[0]) and torch.equal(e.ring._values[:m], want[1])


@pytest.mark.parametrize("d,h,qh", [(128, 8, 32), (128, 2, 16), (256, 4, 16)])
def test_large_scores_of_ring_tokens_keep_their_differences(d, h, qh, dev):
    """Scores of 1024, 1025 and 1026, exact in fp32: only differences reach an exponential, whose argument below 2 and its
    product with log2(e) are rounded to 2^-23 each, its result to 2^-22.  (Scaled to base 2 first, a score of 1477 is rounded by up
    to 6e-5, and so is every probability.)"""
    from turboquant_b200 import CompressedKVStore, compute_hybrid_attention
    store = CompressedKVStore(d, h, 3, 2, device=dev)
    g = torch.Generator(device=dev).manual_seed(d)
    k, q = torch.zeros(256, h, d, device=dev), torch.zeros(1, qh, d, device=dev)
    k[..., 0], k[..., 1] = 32, torch.randint(0, 3, (256, h), generator=g, device=dev).float()
    q[..., 0], q[..., 1] = 32, 1
    v = torch.randn(256, h, d, generator=g, device=dev)
    for r in (5, 33, 64, 128, 256):
        out = compute_hybrid_attention(q, store, k[:r], v[:r], qh, scale=1.0)
        kk, vv = (t[:r].double().transpose(0, 1).repeat_interleave(qh // h, 0) for t in (k, v))
        want = torch.einsum("thn,hnd->thd", torch.softmax(torch.einsum("thd,hnd->thn", q.double(), kk), -1), vv)
        assert _rel(out, want) <= 2e-6, r


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("d", [128, 256])
def test_recent_tokens_from_any_address(d, dtype, dev):
    """Views that begin, or whose rows begin, beside a 16-byte boundary: the same result as from tensors of their own."""
    from turboquant_b200 import CompressedKVStore, compute_hybrid_attention
    h, qh, r, n = 2, 8, 40, 200
    g = torch.Generator(device=dev).manual_seed(d)
    k, v = (torch.randn(n, h, d, generator=g, device=dev, dtype=torch.bfloat16) for _ in range(2))
    store = CompressedKVStore(d, h, 3, 2, device=dev)
    store.append_chunk(k, v)
    rk, rv = (torch.randn(r, h, d, generator=g, device=dev).to(dtype) for _ in range(2))
    q = torch.randn(1, qh, d, generator=g, device=dev, dtype=torch.bfloat16)

    def moved(t, first, stride):
        flat = torch.zeros(first + r * stride, device=dev, dtype=dtype)
        view = flat.as_strided(t.shape, (stride, d, 1), first)
        view.copy_(t)
        return view

    want = compute_hybrid_attention(q, store, rk, rv, qh)
    one = compute_hybrid_attention(q, store, rk[:1], rv[:1], qh)
    for kf, vf, stride in ((1, 0, h * d), (0, 1, h * d), (3, 3, h * d), (0, 0, h * d + 1), (5, 2, h * d + 2)):
        a, b = moved(rk, kf, stride), moved(rv, vf, stride)
        assert torch.equal(compute_hybrid_attention(q, store, a, b, qh), want), (kf, vf, stride)
        assert torch.equal(compute_hybrid_attention(q, store, a[:1], b[:1], qh), one), (kf, vf, stride)
