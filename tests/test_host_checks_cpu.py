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


def test_scratch_of_the_cache_object_is_sized_by_call():
    cfg, out = _lib.tq_config(128, 3, 2, 32), C.c_size_t(0)
    lib = _lib.lib()

    def size(name, *args):
        rc = getattr(lib, name)(C.byref(cfg), *args, C.byref(out))
        return out.value if rc == 0 else rc

    base = size("tq_cache_scores_workspace_bytes", 1, 1) - 2 * 128 * 4
    assert size("tq_cache_scores_workspace_bytes", 32, 4096) == base + 32 * 4096 * 2 * 128 * 4
    # partial sums: no more than the history dequantised to fp32, whatever the number of queries taken
    for heads, n in ((8, 32768), (1, 128)):
        assert size("tq_cache_attend_workspace_bytes", heads, n, 0, 128) == base + heads * n * 128 * 4
        assert size("tq_cache_attend_workspace_bytes", heads, n, 0, 129) == _lib.TQ_ERR_UNSUPPORTED
    assert size("tq_cache_attend_workspace_bytes", 4097, 128, 0, 1) == _lib.TQ_ERR_UNSUPPORTED     # merge tickets
    assert size("tq_cache_attend_workspace_bytes", 4096, 128, 0, 4) > 0
    both = size("tq_cache_workspace_bytes", 8, 4096, 128, 2)
    assert both == max(size("tq_cache_scores_workspace_bytes", 8, 2), size("tq_cache_attend_workspace_bytes", 8, 4096, 128, 2))
    assert size("tq_cache_workspace_bytes", 8, 4096, 0, 4096) == size("tq_cache_scores_workspace_bytes", 8, 4096)
    for bad in ((0, 16, 0, 1), (1, -1, 0, 1), (1, 16, -1, 1), (1, 16, 0, 0)):
        assert size("tq_cache_workspace_bytes", *bad) == _lib.TQ_ERR_SHAPE


def test_the_shared_identity_table_belongs_to_the_device_that_is_current(monkeypatch):
    """A device without an index means the current one at the call, not at the first call."""
    made, now = [], [0]

    def table(n, device):
        made.append(torch.device(device))
        return torch.arange(n, dtype=torch.int32)

    monkeypatch.setattr(E, "_IDENTITY", {})
    monkeypatch.setattr(E, "identity_block_table", table)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: now[0])
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: type("S", (), {"synchronize": lambda self: None})())
    first = E.shared_identity_table(10, "cuda")
    now[0] = 1
    second = E.shared_identity_table(10, torch.device("cuda"))
    assert second is not first and made == [torch.device("cuda", 0), torch.device("cuda", 1)]
    assert E.shared_identity_table(10, torch.device("cuda", 0)) is first and E.shared_identity_table(5, "cuda:1") is second


def test_threads_share_one_set_of_operands(monkeypatch):
    """Two threads that need the operands first at the same time: the structure keeps the addresses of the tensors that the
    object keeps."""
    consts = E.LayerConstants(128, 3, 2, "cpu")
    split, meet = E._split, threading.Barrier(2, timeout=0.5)

    def slow(m, limbs, dtype):
        try:
            meet.wait()        # both threads inside, if both can be
        except threading.BrokenBarrierError:
            pass
        return split(m, limbs, dtype)

    monkeypatch.setattr(E, "_split", slow)
    made, keep = [], E.LayerConstants.__setattr__
    monkeypatch.setattr(E.LayerConstants, "__setattr__", lambda self, k, v: (made.append(v) if k == "rows_limbs" else None, keep(self, k, v))[1])
    threads = [threading.Thread(target=consts.ensure_rows) for _ in range(2)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert len(made) == 1
    for i in range(2):
        assert [consts.c.rows_pi[i], consts.c.rows_m[i], consts.c.rows_s[i]] == [x[i].data_ptr() for x in consts.rows_limbs]


@pytest.mark.parametrize("row,top,taken", [(1.0, 0.2, True), (7.9, 0.2, True), (8.1, 0.2, False), (1.0, 6.9, True), (1.0, 7.1, False)])
def test_operands_of_the_wide_store_keep_residuals_inside_fp16(row, top, taken):
    """Residuals are carried 4096 times: |u| |row of Pi| + |centroid| + what E adds must stay below 65504 / 4096."""
    unit = E.LayerConstants(256, 4, 2, "cpu")
    pi = unit.Pi / unit.Pi.norm(dim=1, keepdim=True) * row
    cents = torch.linspace(-top, top, 8)
    bounds = torch.cat((torch.tensor([-10.0 * top]), (cents[1:] + cents[:-1]) / 2, torch.tensor([10.0 * top])))
    consts = E.LayerConstants(256, 4, 2, "cpu", Pi=pi, centroids=cents, boundaries=bounds)
    assert (consts.rows_limbs is not None) == taken and (consts.c.rows_pi[0] is not None) == taken
    if taken:
        assert (row * (1 + 2 ** -8 + 2 ** -9) * (1 + 2 ** -8) + top) * 4096 < 65504
