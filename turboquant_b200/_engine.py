"""Device-side state shared by the host classes: per-layer constants, block
pools, workspaces, and thin wrappers around the C entry points.

PyTorch is used for device memory and streams only; all arithmetic of the
store and read paths runs in the CUDA library.
"""

from __future__ import annotations

import ctypes as C
import itertools
import math
import threading
from typing import Optional

import torch

from . import _lib
from ._lib import TQ_BF16, TQ_BLOCK_TOKENS, TQ_F16, TQ_F32, check, host, lib
from .codebook import get_codebook_tensors
from .rotation import generate_qjl_matrix, generate_rotation_matrix

_DTYPES = {torch.float32: TQ_F32, torch.bfloat16: TQ_BF16, torch.float16: TQ_F16}


def dtype_code(dt: torch.dtype) -> int:
    try:
        return _DTYPES[dt]
    except KeyError:
        raise TypeError(f"unsupported dtype {dt}; use float32, bfloat16 or float16") from None


def stream_ptr(device) -> int:
    return torch.cuda.current_stream(device).cuda_stream


def require_cuda(t: torch.Tensor, name: str) -> None:
    if not t.is_cuda:
        raise RuntimeError(f"{name} must be a CUDA tensor: this package has no CPU path")


def get_layout(head_dim: int, key_bits: int, value_bits: int, group_size: int = 32) -> _lib.tq_layout:
    cfg = _lib.tq_config(head_dim, key_bits, value_bits, group_size)
    out = _lib.tq_layout()
    check(lib().tq_get_layout(C.byref(cfg), C.byref(out)), "tq_get_layout")
    return out


def _split(m: torch.Tensor, n_limbs: int, dtype: torch.dtype) -> list[torch.Tensor]:
    """m (fp64) as a sum of limbs of `dtype`, largest first."""
    limbs, rest = [], m.clone()
    for _ in range(n_limbs):
        limb = rest.to(torch.float32).to(dtype)
        limbs.append(limb)
        rest = rest - limb.to(torch.float64)
    return limbs


def _split_bf16(m: torch.Tensor, n_limbs: int) -> list[torch.Tensor]:
    return _split(m, n_limbs, torch.bfloat16)


_ROWS_LOCK = threading.Lock()


class LayerConstants:
    """Pi, S, the code book and the C struct that carries them (one per layer and shape).

    Seeds follow the reference: Pi from `seed`, S from `seed + 1000`
    (quantizer.py:208), `seed = 42 + 7 * layer_idx` for a layer (store.py:56).
    """

    def __init__(self, head_dim: int, key_bits: int, value_bits: int, device, seed: int = 42,
                 group_size: int = 32, Pi: Optional[torch.Tensor] = None, S: Optional[torch.Tensor] = None,
                 centroids: Optional[torch.Tensor] = None, boundaries: Optional[torch.Tensor] = None,
                 tensor_core_store: bool = True):
        self.head_dim, self.key_bits, self.value_bits = head_dim, key_bits, value_bits
        self.group_size = group_size
        self.device = torch.device(device)
        self.cfg = _lib.tq_config(head_dim, key_bits, value_bits, group_size)
        self.layout = get_layout(head_dim, key_bits, value_bits, group_size)
        mse_bits = key_bits - 1
        pi = generate_rotation_matrix(head_dim, "cpu", seed=seed) if Pi is None else Pi.detach().float().cpu()
        s = generate_qjl_matrix(head_dim, "cpu", seed=seed + 1000) if S is None else S.detach().float().cpu()
        if centroids is None or boundaries is None:
            centroids, boundaries = get_codebook_tensors(head_dim, mse_bits, "cpu")
        self.centroids_cpu = centroids.detach().float().cpu()
        self.boundaries_cpu = boundaries.detach().float().cpu()
        dev = self.device
        self.Pi = pi.contiguous().to(dev)
        self.PiT = pi.T.contiguous().to(dev)
        self.S = s.contiguous().to(dev)
        self.ST = s.T.contiguous().to(dev)
        self.centroids = self.centroids_cpu.to(dev)
        self.boundaries = self.boundaries_cpu.to(dev)
        self.qjl_scale = math.sqrt(math.pi / 2.0) / head_dim
        # operands of the tensor-core store kernel: Pi as three bf16 limbs and
        # M = S Pi^T (the QJL projection applied in rotated space) as two
        m = s.double() @ pi.double().T
        self.pi_limbs = [t.contiguous().to(dev) for t in _split_bf16(pi.double(), 3)]
        self.m_limbs = [t.contiguous().to(dev) for t in _split_bf16(m, 2)]
        # and of the tensor-core query preparation: S as two bf16 limbs (Pi's first two serve there too)
        self.s_limbs = [t.contiguous().to(dev) for t in _split_bf16(s.double(), 2)]

        c = _lib.tq_consts()
        c.cfg = self.cfg
        c.pi, c.pi_t = self.Pi.data_ptr(), self.PiT.data_ptr()
        c.s, c.s_t = self.S.data_ptr(), self.ST.data_ptr()
        n_cent = 1 << mse_bits
        for i in range(n_cent):
            c.centroids[i] = float(self.centroids_cpu[i])
        interior = self.boundaries_cpu[1:-1]
        for i in range(n_cent - 1):
            c.boundaries[i] = float(interior[i])
        c.qjl_scale = self.qjl_scale
        # without the split operands tq_store always runs its fp32 kernel
        for i in range(3):
            c.pi_limbs[i] = self.pi_limbs[i].data_ptr() if tensor_core_store else None
        for i in range(2):
            c.m_limbs[i] = self.m_limbs[i].data_ptr() if tensor_core_store else None
            c.s_limbs[i] = self.s_limbs[i].data_ptr() if tensor_core_store else None
        self.rows_limbs = None
        if tensor_core_store and head_dim == 256 and (key_bits, value_bits) != (3, 2):
            # the wide records' store keeps 22 bits of Pi and M; its residuals must stay in fp16's range
            if float(pi.norm(dim=1).max()) < 8 and float(self.centroids_cpu.abs().max()) < 7:
                self.rows_limbs = self._fp16_limbs(pi.double() * 64.0, m)
                for i in range(2 if self.rows_limbs else 0):
                    c.rows_pi[i], c.rows_m[i] = (x[i].data_ptr() for x in self.rows_limbs)
        self.c = c
        self.addr = C.addressof(c)     # what the native host path passes on

    def _fp16_limbs(self, *mats: torch.Tensor) -> list:
        """Each matrix as two fp16 limbs on the device; nothing where one leaves fp16's range (a caller's own S may be
        anything)."""
        if not all(bool(t.abs().max() < 60000.0) for t in mats):
            return []
        return [[t.contiguous().to(self.device) for t in _split(x, 2, torch.float16)] for x in mats]

    def ensure_rows(self) -> None:
        """Operands of the kernels on plain rows (64 Pi, M = S Pi^T and S as two fp16 limbs each): only the quantiser
        objects use them, which call this before their first launch."""
        if self.rows_limbs is not None or self.head_dim != 128:
            return
        with _ROWS_LOCK:   # one set per object: the structure holds the addresses of the tensors that rows_limbs keeps
            if self.rows_limbs is not None:
                return
            pi, s = self.Pi.cpu().double(), self.S.cpu().double()
            limbs = self._fp16_limbs(pi * 64.0, s @ pi.T, s)
            for i in range(2 if limbs else 0):
                self.c.rows_pi[i], self.c.rows_m[i], self.c.rows_s[i] = (x[i].data_ptr() for x in limbs)
            self.rows_limbs = limbs

    @property
    def block_bytes(self) -> int:
        return self.layout.block_bytes

    @property
    def bytes_per_token(self) -> int:
        return self.layout.bytes_per_token


class BlockPool:
    """A pool of block records for `num_kv_heads` heads (uint8 device tensor)."""

    def __init__(self, consts: LayerConstants, num_kv_heads: int, num_blocks: int, zeroed: bool = True):
        """zeroed=False: for a pool whose blocks are all written before any is read."""
        self._alloc = torch.zeros if zeroed else torch.empty
        self.consts = consts
        self.num_kv_heads = num_kv_heads
        self.num_blocks = 0
        self.data = torch.empty(0, dtype=torch.uint8, device=consts.device)
        self.c = _lib.tq_pool()
        self.addr = C.addressof(self.c)     # stays valid: the structure is updated in place
        self.resize(max(1, num_blocks))

    def resize(self, num_blocks: int) -> None:
        """Grow (never shrink) to `num_blocks`, keeping existing records."""
        if num_blocks <= self.num_blocks:
            return
        per_block = self.num_kv_heads * self.consts.block_bytes
        new = self._alloc(num_blocks * per_block, dtype=torch.uint8, device=self.consts.device)
        if self.num_blocks:
            new[: self.num_blocks * per_block].copy_(self.data)
        self.data, self.num_blocks = new, num_blocks
        self.c.base, self.c.num_blocks, self.c.num_kv_heads = self.data.data_ptr(), num_blocks, self.num_kv_heads

    def nbytes(self) -> int:
        return self.data.numel()

    @classmethod
    def over(cls, consts: LayerConstants, num_kv_heads: int, raw: torch.Tensor) -> "BlockPool":
        """A pool laid over memory somebody else allocated (a serving engine's KV-cache buffer): `raw`
        is a contiguous uint8 device tensor, 16-byte aligned; as many whole blocks as fit are used.
        The pool never grows and never copies."""
        if raw.dtype != torch.uint8 or not raw.is_cuda or not raw.is_contiguous() or raw.data_ptr() % 16:
            raise ValueError("the pool needs a contiguous, 16-byte aligned uint8 device tensor")
        per_block = num_kv_heads * consts.block_bytes
        n = raw.numel() // per_block
        if n < 1:
            raise ValueError(f"{raw.numel()} bytes hold no block of {per_block} bytes")
        pool = cls.__new__(cls)
        pool.consts, pool.num_kv_heads, pool.num_blocks = consts, num_kv_heads, n
        pool.data = raw.view(-1)[: n * per_block]
        pool.c = _lib.tq_pool(pool.data.data_ptr(), n, num_kv_heads)
        pool.addr = C.addressof(pool.c)
        pool.resize = pool._fixed
        return pool

    def _fixed(self, num_blocks: int) -> None:
        if num_blocks > self.num_blocks:
            raise RuntimeError(f"a pool over engine memory cannot grow ({self.num_blocks} -> {num_blocks} blocks)")


class Workspace:
    """Zero-initialised scratch for tq_decode / tq_scores; grows on demand."""

    def __init__(self, device):
        self.device = torch.device(device)
        self.buf = torch.empty(0, dtype=torch.uint8, device=self.device)

    def ensure(self, nbytes: int) -> None:
        if self.buf.numel() < nbytes:
            self.buf = torch.zeros(nbytes, dtype=torch.uint8, device=self.device)

    def ensure_decode(self, consts: "LayerConstants", b: int, qh: int, h: int, splits: int) -> None:
        """Size the buffer for one tq_decode shape; the library is asked once per shape."""
        key = (consts.head_dim, consts.key_bits, consts.value_bits, b, qh, h, splits)
        need = _DECODE_WS_BYTES.get(key)
        if need is None:
            n = C.c_size_t(0)
            check(lib().tq_decode_workspace_bytes(C.byref(consts.cfg), b, qh, h, splits, C.byref(n)),
                  "tq_decode_workspace_bytes")
            need = _DECODE_WS_BYTES[key] = n.value
        self.ensure(need)

    @property
    def ptr(self) -> int:
        return self.buf.data_ptr()

    @property
    def nbytes(self) -> int:
        return self.buf.numel()

    def status(self) -> int:
        out = C.c_int32(0)
        check(lib().tq_read_status(self.ptr, stream_ptr(self.device), C.byref(out)), "tq_read_status")
        return out.value


_SM_COUNT: dict[int, int] = {}
_DECODE_WS_BYTES: dict[tuple, int] = {}
_CONST_I32: dict[tuple, torch.Tensor] = {}


def const_i32(device, value: int, n: int = 1) -> torch.Tensor:
    """A cached read-only int32 device tensor of `n` copies of `value` (sequence
    and ring lengths handed to the kernels; small values only are cached)."""
    if not 0 <= value <= 4096 or n > 64:
        return torch.full((n,), value, dtype=torch.int32, device=device)
    key = (str(device), value, n)
    t = _CONST_I32.get(key)
    if t is None:
        t = _CONST_I32[key] = torch.full((n,), value, dtype=torch.int32, device=device)
    return t


def sm_count(device) -> int:
    idx = torch.device(device).index or 0
    if idx not in _SM_COUNT:
        _SM_COUNT[idx] = torch.cuda.get_device_properties(idx).multi_processor_count
    return _SM_COUNT[idx]


def choose_splits(batch: int, num_kv_heads: int, max_seq_len: int, sms: int, max_ring_len: int = 0) -> int:
    """Sequence splits per (sequence, kv head) that suit a launch of this shape on `sms` multiprocessors."""
    return lib().tq_decode_splits(batch, num_kv_heads, max_seq_len, max_ring_len, sms)


def store(consts: LayerConstants, pool: BlockPool, key: torch.Tensor, value: torch.Tensor, *,
          stride_token: int, stride_head: int, n_tokens: int, n_heads: int,
          slot_mapping: Optional[torch.Tensor] = None, block_table: Optional[torch.Tensor] = None,
          start_pos: int = 0) -> None:
    require_cuda(key, "key")
    require_cuda(value, "value")
    if key.dtype != value.dtype:
        raise TypeError("key and value must share a dtype")
    check(lib().tq_store(C.byref(consts.c), key.data_ptr(), value.data_ptr(), dtype_code(key.dtype),
                         n_tokens, n_heads, stride_token, stride_head,
                         slot_mapping.data_ptr() if slot_mapping is not None else None,
                         block_table.data_ptr() if block_table is not None else None,
                         start_pos, C.byref(pool.c), stream_ptr(consts.device)), "tq_store")


def store_paged(consts: LayerConstants, pool: BlockPool, key_cache: torch.Tensor, value_cache: torch.Tensor, *,
                src_block_table: torch.Tensor, n_tokens: int, block_table: torch.Tensor, start_pos: int = 0,
                any_width: bool = False) -> bool:
    """Compress the first n_tokens tokens of a sequence held in a paged cache.

    key_cache / value_cache: (num_blocks, block_size, H, D) views (any block / token / head strides, D
    contiguous, same strides for both); src_block_table: int32 device tensor, logical -> physical block.
    Returns False, with nothing launched, when the call does not fit the table-walking tensor-core
    kernel (the caller then gathers the rows and uses `store`).  any_width: take head_dim 256 with 4-bit
    keys or values too, which callers without it may rely on being refused.
    """
    require_cuda(key_cache, "key_cache")
    require_cuda(value_cache, "value_cache")
    if key_cache.dtype != value_cache.dtype or key_cache.shape != value_cache.shape or \
            key_cache.stride() != value_cache.stride() or key_cache.dim() != 4 or key_cache.stride(3) != 1:
        raise ValueError("key_cache and value_cache must be (num_blocks, block_size, H, D) views of one layout")
    if src_block_table.dtype != torch.int32 or not src_block_table.is_cuda or not src_block_table.is_contiguous():
        raise TypeError("src_block_table must be a contiguous int32 device tensor")
    nb, bs, h, _ = key_cache.shape
    if n_tokens > src_block_table.numel() * bs:
        raise ValueError("src_block_table is shorter than n_tokens")
    fn = lib().tq_store_paged_any if any_width else lib().tq_store_paged
    rc = fn(C.byref(consts.c), key_cache.data_ptr(), value_cache.data_ptr(), dtype_code(key_cache.dtype), nb, bs, h,
            key_cache.stride(0), key_cache.stride(1), key_cache.stride(2), src_block_table.data_ptr(), n_tokens,
            block_table.data_ptr(), start_pos, C.byref(pool.c), stream_ptr(consts.device))
    if rc == _lib.TQ_ERR_UNSUPPORTED:
        return False
    check(rc, "tq_store_paged")
    return True


_REPORT_WORDS = 1024
_report_page: Optional[torch.Tensor] = None     # page-locked: a launch may write a word as long as the process lives
_report_ticket = itertools.count(1)
_report_lock = threading.Lock()


class RangeReport:
    """A word of host memory that a launch sets to a number of its own when it meets an index out of range: looked at
    without a synchronisation, so an error shows once the launch has run.  Two launches 1024 apart share a word, and the
    later error then hides the earlier one; neither is taken for the other's."""

    def __init__(self, page: torch.Tensor):
        self.ticket = next(_report_ticket) & 0x7fffffff
        self.address = page.data_ptr() + 4 * (self.ticket % _REPORT_WORDS)
        self._word = C.c_int32.from_address(self.address)

    @property
    def failed(self) -> bool:
        return self._word.value == self.ticket


def range_report() -> Optional[RangeReport]:
    """None while the page would have to be made under stream capture."""
    global _report_page
    if _report_page is None:
        if torch.cuda.is_current_stream_capturing():
            return None
        with _report_lock:
            if _report_page is None:
                _report_page = torch.zeros(_REPORT_WORDS, dtype=torch.int32).pin_memory()
    return RangeReport(_report_page)


def ring_write_paged(ring_k: torch.Tensor, ring_v: torch.Tensor, position: int, key_cache: torch.Tensor, value_cache: torch.Tensor,
                     src_block_table: torch.Tensor, first: int, n: int, report: Optional[RangeReport] = None) -> bool:
    """Tokens [first, first + n) of a sequence in a paged cache ((num_blocks, block_size, H, D) planes of one layout,
    `src_block_table` int32, contiguous) into the ring's buffers from `position` on, in one launch.  False, with nothing
    launched, for tensors that the kernel does not take."""
    nb, bs, h, d = key_cache.shape
    if not (key_cache.is_cuda and ring_k.device == key_cache.device == value_cache.device == src_block_table.device
            and ring_k.dtype == key_cache.dtype == value_cache.dtype and key_cache.dtype in _DTYPES
            and key_cache.stride() == value_cache.stride() and key_cache.shape == value_cache.shape and key_cache.stride(3) == 1
            and min(key_cache.stride()) >= 0 and tuple(ring_k.shape[1:]) == (h, d) and src_block_table.dtype == torch.int32
            and src_block_table.is_contiguous() and first + n <= src_block_table.numel() * bs and position + n <= ring_k.shape[0]):
        return False
    rc = lib().tq_ring_write_paged_reported(
        key_cache.data_ptr(), value_cache.data_ptr(), _DTYPES[key_cache.dtype], nb, bs, h, d, key_cache.stride(0), key_cache.stride(1),
        key_cache.stride(2), src_block_table.data_ptr(), first, n, ring_k.data_ptr(), ring_v.data_ptr(), ring_k.stride(0), position,
        report.address if report else None, report.ticket if report else 0, stream_ptr(ring_k.device))
    if rc in (_lib.TQ_ERR_UNSUPPORTED, _lib.TQ_ERR_ALIGN):
        return False
    check(rc, "tq_ring_write_paged")
    return True


def decode(consts: LayerConstants, pool: BlockPool, ws: Workspace, query: torch.Tensor,
           block_table: torch.Tensor, seq_lens: torch.Tensor, max_seq_len: int, *,
           ring_k: Optional[torch.Tensor] = None, ring_v: Optional[torch.Tensor] = None,
           ring_lens: Optional[torch.Tensor] = None, max_ring_len: int = 0,
           ring_stride_seq: int = 0, ring_stride_token: int = 0, scale: Optional[float] = None,
           min_history: int = 16, num_splits: int = 0, out: Optional[torch.Tensor] = None,
           query_prepared: bool = False, kernel: int = 0, static_scratch: bool = False,
           append_k: Optional[torch.Tensor] = None, append_v: Optional[torch.Tensor] = None) -> torch.Tensor:
    """query (B, Qh, D) -> out (B, Qh, D) in the query dtype.

    static_scratch=True routes through tq_decode_static: no workspace tensor is
    touched, the library's built-in scratch array is used (for callers that
    must not allocate); `ws` may then be None.
    """
    require_cuda(query, "query")
    b, qh, d = query.shape
    query = query.contiguous()
    if out is None:
        out = torch.empty_like(query)
    require_cuda(out, "out")
    if scale is None:
        scale = 1.0 / math.sqrt(d)
    h = pool.num_kv_heads
    splits = num_splits or choose_splits(b, h, max_seq_len, sm_count(consts.device), max_ring_len)
    if not static_scratch:
        ws.ensure_decode(consts, b, qh, h, splits)
    a = _lib.tq_decode_args()
    a.query, a.q_dtype, a.batch, a.num_q_heads = query.data_ptr(), dtype_code(query.dtype), b, qh
    a.block_table = block_table.data_ptr()
    a.block_table_stride = block_table.stride(0) if block_table.dim() == 2 else block_table.numel()
    a.seq_lens, a.max_seq_len, a.min_history = seq_lens.data_ptr(), max_seq_len, min_history
    if ring_k is not None and max_ring_len > 0:
        a.ring_k, a.ring_v = ring_k.data_ptr(), ring_v.data_ptr()
        a.ring_dtype = dtype_code(ring_k.dtype)
        a.ring_lens, a.max_ring_len = ring_lens.data_ptr(), max_ring_len
        a.ring_stride_seq, a.ring_stride_token = ring_stride_seq, ring_stride_token
    a.scale = scale
    a.out, a.num_splits = out.data_ptr(), splits
    a.query_prepared = 1 if query_prepared else 0
    a.kernel = kernel
    if append_k is not None:      # (B, H, D) new exact token per sequence, appended on the device before attending
        a.append_k, a.append_v = append_k.data_ptr(), append_v.data_ptr()
        a.ring_capacity = ring_k.shape[-3]
    if static_scratch:
        check(lib().tq_decode_static(C.byref(consts.c), C.byref(pool.c), C.byref(a), stream_ptr(consts.device)),
              f"tq_decode_static (built-in scratch of {lib().tq_decode_static_scratch_bytes()} bytes)")
        return out
    a.workspace, a.workspace_bytes = ws.ptr, ws.nbytes
    check(lib().tq_decode(C.byref(consts.c), C.byref(pool.c), C.byref(a), stream_ptr(consts.device)), "tq_decode")
    return out


def scores(consts: LayerConstants, pool: BlockPool, ws: Workspace, block_table: torch.Tensor, n_tokens: int,
           query: torch.Tensor) -> torch.Tensor:
    """query (H, n_q, D) -> unscaled logits (H, n_q, n_tokens) fp32."""
    require_cuda(query, "query")
    h, n_q, d = query.shape
    query = query.contiguous()
    logits = torch.empty(h, n_q, n_tokens, dtype=torch.float32, device=query.device)
    need = C.c_size_t(0)
    check(lib().tq_scores_workspace_bytes(C.byref(consts.cfg), h * n_q, C.byref(need)), "tq_scores_workspace_bytes")
    ws.ensure(need.value)
    check(lib().tq_scores(C.byref(consts.c), C.byref(pool.c), block_table.data_ptr(), n_tokens, query.data_ptr(),
                          dtype_code(query.dtype), n_q, logits.data_ptr(), ws.ptr, ws.nbytes,
                          stream_ptr(consts.device)), "tq_scores")
    return logits


class PlaneSet:
    """Flat planes (H, capacity, ...) on the device plus their C descriptor."""

    def __init__(self, consts: LayerConstants, num_kv_heads: int, capacity: int, zeroed: bool = True):
        """zeroed=False: for planes that a conversion fills completely."""
        lay, dev = consts.layout, consts.device
        h, n = num_kv_heads, max(1, capacity)
        new = torch.zeros if zeroed else torch.empty
        self.mse_indices = new(h, n, lay.kcode_row, dtype=torch.uint8, device=dev)
        self.qjl_signs = new(h, n, lay.ksign_row, dtype=torch.uint8, device=dev)
        self.norms = new(h, n, dtype=torch.float16, device=dev)
        self.residual_norms = new(h, n, dtype=torch.float16, device=dev)
        self.v_data = new(h, n, lay.vcode_row, dtype=torch.uint8, device=dev)
        self.v_scales = new(h, n, lay.n_groups, dtype=torch.float16, device=dev)
        self.v_zeros = new(h, n, lay.n_groups, dtype=torch.float16, device=dev)
        self.capacity = n
        self.c = _lib.tq_planes(self.mse_indices.data_ptr(), self.qjl_signs.data_ptr(), self.norms.data_ptr(),
                                self.residual_norms.data_ptr(), self.v_data.data_ptr(), self.v_scales.data_ptr(),
                                self.v_zeros.data_ptr(), n)

    @classmethod
    def from_tensors(cls, consts, mse_indices, qjl_signs, norms, residual_norms, v_data, v_scales, v_zeros):
        h, n = mse_indices.shape[0], mse_indices.shape[1]
        ps = cls(consts, h, n)
        dev = consts.device
        ps.mse_indices.copy_(mse_indices.to(dev))
        ps.qjl_signs.copy_(qjl_signs.to(dev))
        ps.norms.copy_(norms.to(dev).to(torch.float16))
        ps.residual_norms.copy_(residual_norms.to(dev).to(torch.float16))
        ps.v_data.copy_(v_data.to(dev))
        ps.v_scales.copy_(v_scales.to(dev).to(torch.float16))
        ps.v_zeros.copy_(v_zeros.to(dev).to(torch.float16))
        return ps


def pool_to_planes(consts: LayerConstants, pool: BlockPool, block_table: torch.Tensor, n_tokens: int) -> PlaneSet:
    ps = PlaneSet(consts, pool.num_kv_heads, n_tokens, zeroed=n_tokens < 1)
    check(lib().tq_pool_to_planes(C.byref(consts.cfg), C.byref(pool.c), block_table.data_ptr(), n_tokens,
                                  C.byref(ps.c), stream_ptr(consts.device)), "tq_pool_to_planes")
    return ps


def planes_to_pool(consts: LayerConstants, planes: PlaneSet, n_tokens: int, pool: BlockPool,
                   block_table: torch.Tensor, start_pos: int = 0) -> None:
    check(lib().tq_planes_to_pool(C.byref(consts.cfg), C.byref(planes.c), n_tokens, block_table.data_ptr(),
                                  start_pos, C.byref(pool.c), stream_ptr(consts.device)), "tq_planes_to_pool")


def dequant_keys(consts: LayerConstants, pool: BlockPool, block_table: torch.Tensor, n_tokens: int,
                 with_qjl: bool = True) -> torch.Tensor:
    out = torch.empty(pool.num_kv_heads, n_tokens, consts.head_dim, dtype=torch.float32, device=consts.device)
    check(lib().tq_dequant_keys(C.byref(consts.c), C.byref(pool.c), block_table.data_ptr(), n_tokens,
                                1 if with_qjl else 0, out.data_ptr(), stream_ptr(consts.device)), "tq_dequant_keys")
    return out


def dequant_values(consts: LayerConstants, pool: BlockPool, block_table: torch.Tensor, n_tokens: int) -> torch.Tensor:
    out = torch.empty(pool.num_kv_heads, n_tokens, consts.head_dim, dtype=torch.float32, device=consts.device)
    check(lib().tq_dequant_values(C.byref(consts.cfg), C.byref(pool.c), block_table.data_ptr(), n_tokens,
                                  out.data_ptr(), stream_ptr(consts.device)), "tq_dequant_values")
    return out


def taken(result, what: str):
    """What a call of the native host path returned: its tensors, None where it left the call to the general way; raises on a
    status."""
    if type(result) is int:
        check(result, what)
    return result


def _float_code(t: torch.Tensor) -> Optional[int]:
    return _DTYPES.get(t.dtype)


def rows_quantize_keys(consts: LayerConstants, x: torch.Tensor):
    """(n, D) rows -> (codes, sign bits, norms in x's dtype, residual norms fp32), or None where the rows kernel does not
    take them (head_dim 256, no split operands, unaligned rows)."""
    if consts.head_dim != 128 or not x.is_cuda or x.dtype not in _DTYPES or x.stride(1) != 1:
        return None
    n, lay, dev = x.shape[0], consts.layout, x.device
    codes = torch.empty(n, lay.kcode_row, dtype=torch.uint8, device=dev)
    signs = torch.empty(n, lay.ksign_row, dtype=torch.uint8, device=dev)
    norms = torch.empty(n, dtype=x.dtype, device=dev)
    rnorms = torch.empty(n, dtype=torch.float32, device=dev)
    rc = lib().tq_rows_quantize_keys(consts.addr, x.data_ptr(), _DTYPES[x.dtype], n, x.stride(0), codes.data_ptr(), signs.data_ptr(),
                                     norms.data_ptr(), _DTYPES[x.dtype], rnorms.data_ptr(), TQ_F32, stream_ptr(dev))
    if rc in (_lib.TQ_ERR_UNSUPPORTED, _lib.TQ_ERR_ALIGN, _lib.TQ_ERR_SHAPE):
        return None
    check(rc, "tq_rows_quantize_keys")
    return codes, signs, norms, rnorms


def key_planes_fit(consts: LayerConstants, n: int, codes, signs, norms, rnorms) -> bool:
    """Whether contiguous planes hold n keys of this configuration, byte planes as bytes, all on one device: what the kernels
    on plain rows take on trust.  signs / rnorms may both be None."""
    lay = consts.layout
    planes = [(codes, n * lay.kcode_row, True), (norms, n, False)]
    if signs is not None or rnorms is not None:
        planes += [(signs, n * lay.ksign_row, True), (rnorms, n, False)]
    return all(t is not None and t.device == codes.device and t.numel() == count and t.is_contiguous()
               and (t.dtype == torch.uint8 if is_bytes else t.dtype in _DTYPES) for t, count, is_bytes in planes)


def value_planes_fit(n: int, d: int, bits: int, data, scales, zeros) -> bool:
    """The same for value codes, scales and zero points of n rows of d values."""
    return (data.dtype == torch.uint8 and data.numel() == n * d * bits // 8 and scales.dtype in _DTYPES and zeros.dtype == scales.dtype
            and all(t.device == data.device and t.numel() == n * (d // 32) for t in (scales, zeros))
            and all(t.is_contiguous() for t in (data, scales, zeros)))


def rows_dequantize_keys(consts: LayerConstants, codes, signs, norms, rnorms) -> Optional[torch.Tensor]:
    """Contiguous key planes (n, ...) -> (n, D) fp32; signs / rnorms None: the MSE part alone.  None where the rows kernel
    does not take them."""
    n = norms.numel()
    if not codes.is_cuda or not key_planes_fit(consts, n, codes, signs, norms, rnorms):
        return None
    out = torch.empty(n, consts.head_dim, dtype=torch.float32, device=codes.device)
    rc = lib().tq_rows_dequantize_keys(consts.addr, codes.data_ptr(), signs.data_ptr() if signs is not None else None, norms.data_ptr(),
                                       _float_code(norms), rnorms.data_ptr() if rnorms is not None else None,
                                       _float_code(rnorms) if rnorms is not None else TQ_F32, n, 0 if signs is None else 1,
                                       out.data_ptr(), stream_ptr(codes.device))
    if rc in (_lib.TQ_ERR_UNSUPPORTED, _lib.TQ_ERR_ALIGN):
        return None
    check(rc, "tq_rows_dequantize_keys")
    return out


def rows_scores(consts: LayerConstants, ws: "Workspace", codes, signs, norms, rnorms, heads: int, n: int,
                query: torch.Tensor) -> Optional[torch.Tensor]:
    """Key planes (heads, n, ...) and query (heads, n_q, D) -> unscaled logits (heads, n_q, n) fp32, or None."""
    if not codes.is_cuda or query.device != codes.device or _float_code(query) is None or \
            not key_planes_fit(consts, heads * n, codes, signs, norms, rnorms) or query.shape[::2] != (heads, consts.head_dim):
        return None
    n_q = query.shape[1]
    need = C.c_size_t(0)
    check(lib().tq_scores_workspace_bytes(C.byref(consts.cfg), heads * n_q, C.byref(need)), "tq_scores_workspace_bytes")
    ws.ensure(need.value)
    logits = torch.empty(heads, n_q, n, dtype=torch.float32, device=codes.device)
    rc = lib().tq_rows_scores(consts.addr, codes.data_ptr(), signs.data_ptr(), norms.data_ptr(), _float_code(norms), rnorms.data_ptr(),
                              _float_code(rnorms), heads, n, query.data_ptr(), _float_code(query), n_q, logits.data_ptr(), ws.ptr,
                              ws.nbytes, stream_ptr(codes.device))
    if rc in (_lib.TQ_ERR_UNSUPPORTED, _lib.TQ_ERR_ALIGN):
        return None
    check(rc, "tq_rows_scores")
    return logits


def rows_quantize_values(v: torch.Tensor, bits: int):
    """(n, D) rows -> (codes, scales, zero points in v's dtype), or None (unaligned rows)."""
    n, d = v.shape
    g = d // 32
    data = torch.empty(n, d * bits // 8, dtype=torch.uint8, device=v.device)
    sz = torch.empty(2, n, g, dtype=v.dtype, device=v.device)
    rc = lib().tq_rows_quantize_values(v.data_ptr(), dtype_code(v.dtype), n, d, v.stride(0), bits, data.data_ptr(), sz[0].data_ptr(),
                                       sz[1].data_ptr(), stream_ptr(v.device))
    if rc in (_lib.TQ_ERR_ALIGN, _lib.TQ_ERR_SHAPE):
        return None
    check(rc, "tq_rows_quantize_values")
    return data, sz[0], sz[1]


def rows_dequantize_values(data: torch.Tensor, scales: torch.Tensor, zeros: torch.Tensor, bits: int, d: int) -> Optional[torch.Tensor]:
    """Contiguous value planes -> (n, D) fp32, or None."""
    n = data.numel() // data.shape[-1]
    if not data.is_cuda or not value_planes_fit(n, d, bits, data, scales, zeros):
        return None
    out = torch.empty(n, d, dtype=torch.float32, device=data.device)
    rc = lib().tq_rows_dequantize_values(data.data_ptr(), scales.data_ptr(), zeros.data_ptr(), _float_code(scales), n, d, bits,
                                         out.data_ptr(), stream_ptr(data.device))
    if rc == _lib.TQ_ERR_ALIGN:
        return None
    check(rc, "tq_rows_dequantize_values")
    return out


def _cache_call(fn, consts, pool, ws, block_table, n, x, buf, *scale) -> Optional[torch.Tensor]:
    """One of the cache object's native calls; a second time on contiguous copies where the strides were the reason."""
    out = fn(consts.addr, pool.addr, ws, block_table, n, x, buf, *scale)
    if out is None:
        args = x.contiguous(), buf.contiguous() if buf is not None else None
        if args[0] is not x or args[1] is not buf:
            out = fn(consts.addr, pool.addr, ws, block_table, n, *args, *scale)
    return None if out is NotImplemented else taken(out, fn.__name__)


def cache_scores(consts: LayerConstants, pool: BlockPool, ws: Workspace, block_table: torch.Tensor, n: int, query: torch.Tensor,
                 buf: Optional[torch.Tensor], scale: float) -> Optional[torch.Tensor]:
    """query (b, h, n_q, D) -> scaled logits (b, h, n_q, n + buffer) fp32, or None where the kernel does not apply."""
    return _cache_call(host().cache_scores, consts, pool, ws, block_table, n, query, buf, scale)


def cache_attend(consts: LayerConstants, pool: BlockPool, ws: Workspace, block_table: torch.Tensor, n: int, weights: torch.Tensor,
                 buf: Optional[torch.Tensor]) -> Optional[torch.Tensor]:
    """weights (b, h, n_q, n + buffer) -> (b, h, n_q, D) fp32, or None where the kernel does not apply."""
    return _cache_call(host().cache_attend, consts, pool, ws, block_table, n, weights, buf)


def identity_block_table(n_blocks: int, device) -> torch.Tensor:
    return torch.arange(max(1, n_blocks), dtype=torch.int32, device=device)


_IDENTITY: dict[str, torch.Tensor] = {}
_IDENTITY_ENTRIES = 65536


def shared_identity_table(n_blocks: int, device) -> torch.Tensor:
    """A read-only identity table of at least `n_blocks` entries: one of 64 K entries per device, made once and never
    replaced, so that any stream may read it; a table of its own beyond that.  A device without an index means the
    current one, at this call."""
    device = torch.device(device)
    if device.index is None:
        device = torch.device(device.type, torch.cuda.current_device())
    key = str(device)
    t = _IDENTITY.get(key)
    if n_blocks > _IDENTITY_ENTRIES or (t is None and torch.cuda.is_current_stream_capturing()):
        return identity_block_table(n_blocks, device)
    if t is None:
        t = identity_block_table(_IDENTITY_ENTRIES, device)
        torch.cuda.current_stream(t.device).synchronize()
        t = _IDENTITY.setdefault(key, t)
    return t


def blocks_for(n_tokens: int) -> int:
    return (n_tokens + TQ_BLOCK_TOKENS - 1) // TQ_BLOCK_TOKENS


def pack_stage(consts: LayerConstants, y: torch.Tensor, projected: torch.Tensor):
    """Integer stages only: rotated vectors -> packed codes, projections -> packed signs."""
    require_cuda(y, "y")
    d = consts.head_dim
    y2 = y.reshape(-1, d).float().contiguous()
    p2 = projected.reshape(-1, d).float().contiguous()
    n = y2.shape[0]
    codes = torch.empty(n, consts.layout.kcode_row, dtype=torch.uint8, device=y.device)
    signs = torch.empty(n, d // 8, dtype=torch.uint8, device=y.device)
    check(lib().tq_pack_stage(C.byref(consts.c), y2.data_ptr(), p2.data_ptr(), n, codes.data_ptr(),
                              signs.data_ptr(), stream_ptr(consts.device)), "tq_pack_stage")
    return codes.reshape(*y.shape[:-1], -1), signs.reshape(*y.shape[:-1], -1)


def prefill_attention_supported(query: torch.Tensor, key: torch.Tensor, value: torch.Tensor) -> bool:
    """Whether `prefill_attention` takes these tensors (CUDA, bf16 / fp16, head_dim 128 or 256, 16-byte
    aligned rows); otherwise the caller keeps its own attention."""
    return (query.is_cuda and key.is_cuda and value.is_cuda and query.dtype in (torch.bfloat16, torch.float16)
            and key.dtype == query.dtype and value.dtype == query.dtype and query.dim() == 3 and key.dim() == 3
            and query.shape[-1] in (128, 256) and key.shape == value.shape and key.shape[-1] == query.shape[-1]
            and query.shape[1] % key.shape[1] == 0 and key.shape[0] == query.shape[0])


def prefill_attention(query: torch.Tensor, key: torch.Tensor, value: torch.Tensor, scale: Optional[float] = None,
                      out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Causal attention of a sequence over itself: query (n, Qh, D), key / value (n, H, D) -> (n, Qh, D)."""
    if not prefill_attention_supported(query, key, value):
        raise ValueError("prefill_attention needs CUDA bf16/fp16 tensors (n, heads, 128 or 256)")

    def rows(t):   # D contiguous, 16-byte aligned rows, token stride >= head stride
        ok = t.stride(2) == 1 and t.stride(0) % 8 == 0 and t.stride(1) % 8 == 0 and t.data_ptr() % 16 == 0 \
            and (t.stride(0) >= t.stride(1) or t.shape[1] == 1) and t.stride(1) >= t.shape[2]
        return t if ok else t.contiguous()

    q, k, v = rows(query), rows(key), rows(value)
    if k.stride() != v.stride():
        k, v = k.contiguous(), v.contiguous()
    n, qh, d = q.shape
    if out is None:
        out = torch.empty((n, qh, d), dtype=q.dtype, device=q.device)
    if scale is None:
        scale = 1.0 / math.sqrt(d)
    check(lib().tq_prefill_attention(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), dtype_code(q.dtype),
                                     n, qh, k.shape[1], d, q.stride(0), q.stride(1), k.stride(0), k.stride(1),
                                     out.stride(0), out.stride(1), float(scale), stream_ptr(q.device)),
          "tq_prefill_attention")
    return out


def prefill_attention_status() -> int:
    """Status word of the prefill attention kernel (0 = fine); synchronises the device."""
    out = C.c_int32(0)
    check(lib().tq_prefill_attention_read_status(C.byref(out)), "tq_prefill_attention_read_status")
    return out.value


def store_status() -> int:
    """Status word of the tensor-core store kernel (0 = fine); synchronises the device."""
    out = C.c_int32(0)
    check(lib().tq_store_read_status(C.byref(out)), "tq_store_read_status")
    return out.value
