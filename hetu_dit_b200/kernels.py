"""Tensor-level entry points over the C ABI (torch is used for device memory and streams only)."""
import contextlib
import ctypes
import functools
import os

import torch
from torch.nn.modules import module as _all_modules

from . import _C

_DTYPE_CODE = {torch.bfloat16: _C.HDIT_BF16, torch.float16: _C.HDIT_FP16}

# Launch accounting for benchmarks: how many kernels of this library were enqueued, and
# (optionally) CUDA-event pairs around every attention launch on its own stream.
_launches = 0
_attn_timing = False
_attn_events = []


def reset_counters():
    global _launches
    _launches = 0
    _attn_events.clear()


def launch_count() -> int:
    return _launches


def enable_attn_timing(on: bool):
    global _attn_timing
    _attn_timing = bool(on)


def attn_timing_summary():
    """Mean device time of the attention launches recorded since reset_counters() (synchronises)."""
    torch.cuda.synchronize()
    ms = [a.elapsed_time(b) for a, b, _ in _attn_events]
    return {"count": len(ms), "mean_ms": (sum(ms) / len(ms)) if ms else None, "min_ms": min(ms) if ms else None,
            "total_ms": sum(ms), "flops": float(sum(f for _, _, f in _attn_events))}


def _count(n=1):
    global _launches
    _launches += n


_NO_SWITCH = contextlib.nullcontext()


_INDEXED = {torch.device("cuda", i): i for i in range(64)}  # looking a device up costs less than asking for its type


def _cuda_index(device):
    """Index of a CUDA device given as a torch.device, a string, an integer or None; the current one's where it names
    none. Any other kind of device is refused: the addresses of its tensors are not the GPU's."""
    if isinstance(device, int):  # -1 is the current device, as for torch.cuda.device()
        return torch.cuda.current_device() if device < 0 else device
    device = torch.device("cuda" if device is None else device)
    if device.type != "cuda":
        raise ValueError(f"expected a cuda device, got {device}")
    return torch.cuda.current_device() if device.index is None else device.index


def _on(device):
    """A context in which `device` is the current one; entering it costs nothing when it already is, as in a process
    that drives one GPU."""
    index = _INDEXED.get(device)
    if index is None:
        index = _cuda_index(device)
    return _NO_SWITCH if index == torch.cuda.current_device() else torch.cuda.device(index)


def _stream_ptr(device):
    """The current stream of `device` as an address, without a Stream object around it (1.5 us of a 14 us call)."""
    index = _INDEXED.get(device)
    return torch._C._cuda_getCurrentRawStream(_cuda_index(device) if index is None else index)


def _fill_seg(seg, t):
    if t.dim() != 4:
        raise ValueError(f"expected a (B, S, H, D) tensor, got shape {tuple(t.shape)}")
    if t.stride(3) != 1 and t.shape[3] != 1:
        raise ValueError("the head dimension must be contiguous")
    seg.ptr, seg.len = t.data_ptr(), t.shape[1]
    seg.stride_b, seg.stride_s, seg.stride_h = t.stride()[:3]


def attn_fwd(
    q_segs,
    k_segs,
    v_segs,
    *,
    softmax_scale=None,
    out=None,
    return_lse=False,
    mode=_C.ATTN_FINAL,
    acc_out=None,
    acc_lse=None,
    kv_split=None,
    kv_interleave=0,
    out_dsts=None,
    q_rows_per_dst=None,
    q_dst_row0=None,
    wait_flags=None,
):
    """softmax(Q K^T * scale) V over segment lists, (B, S, H, D) layout.

    q_segs / k_segs / v_segs are lists of tensors that are logically concatenated
    along S (no copy is made). Returns `out` of shape (B, sum Sq, H, D) in the input
    dtype (and the (B, H, Sq) fp32 log-sum-exp when return_lse is set). In the
    PARTIAL modes nothing is returned; the fp32 running result lives in acc_out /
    acc_lse, which a later MERGE call combines with its own block by log-sum-exp.

    kv_split (FINAL mode only): number of CTAs that share one query tile pair, each over its own
    range of KV blocks, merged by a second small kernel. None picks it from the grid size: a head-
    and sequence-sharded call can have fewer tile pairs than the GPU has SMs.
    kv_interleave: 0 lets the library decide, 1 forbids, 2 forces the mode in which a CTA owns one query tile
    and its two halves take the even and odd KV blocks (merged in shared memory; for small grids).

    out_dsts (a RawDst: device addresses + (b, s, h) element strides): scatter the result rows over these
    buffers instead of returning one tensor -- row r of query segment s goes to destination
    r // q_rows_per_dst[s] at row q_dst_row0[s] + r % q_rows_per_dst[s], or to every destination at row
    q_dst_row0[s] + r when q_rows_per_dst[s] is 0. With the Ulysses peers' output buffers as destinations this
    is the reverse all-to-all done by the attention epilogue. Returns None (or the lse) in that case.

    wait_flags (a FlagWait): flags in this rank's memory that the peers' exchange kernels bump; the kernel's
    loader waits for them before its first load (the barrier after the head exchange, folded into attention).
    """
    q0 = q_segs[0]
    if not q0.is_cuda:
        raise RuntimeError("hetu_dit_b200 kernels need CUDA tensors; there is no CPU path")
    if q0.dtype not in _DTYPE_CODE:
        raise TypeError(f"unsupported dtype {q0.dtype}")
    if len(k_segs) != len(v_segs):
        raise ValueError("k and v segment lists differ in length")
    B, _, H, D = q0.shape
    sq = sum(int(t.shape[1]) for t in q_segs)
    a = _C.AttnArgs()
    a.dtype = _DTYPE_CODE[q0.dtype]
    a.mode = mode
    a.batch, a.heads, a.head_dim = B, H, D
    a.n_q_seg, a.n_kv_seg = len(q_segs), len(k_segs)
    a.softmax_scale = float(softmax_scale) if softmax_scale is not None else 0.0
    if len(q_segs) > _C.HDIT_MAX_Q_SEG or len(k_segs) > _C.HDIT_MAX_KV_SEG:
        raise ValueError("too many segments")
    for i, t in enumerate(q_segs):
        _fill_seg(a.q[i], t)
    for i, (k, v) in enumerate(zip(k_segs, v_segs)):
        _fill_seg(a.k[i], k)
        _fill_seg(a.v[i], v)
    writes_out = mode in (_C.ATTN_FINAL, _C.ATTN_MERGE_FINAL)
    lse = None
    a.kv_interleave = int(kv_interleave)
    if writes_out and out_dsts is not None:
        a.n_out_dst = len(out_dsts)
        for i, ptr in enumerate(out_dsts.ptrs):
            a.out_dst[i] = ptr
        a.out_stride_b, a.out_stride_s, a.out_stride_h = out_dsts.strides
        for i in range(len(q_segs)):
            a.q_rows_per_dst[i] = int(q_rows_per_dst[i])
            a.q_dst_row0[i] = int(q_dst_row0[i])
        if return_lse:
            lse = torch.empty((B, H, sq), dtype=torch.float32, device=q0.device)
            a.lse = lse.data_ptr()
    elif writes_out:
        if out is None:
            out = torch.empty((B, sq, H, D), dtype=q0.dtype, device=q0.device)
        a.out = out.data_ptr()
        a.out_stride_b, a.out_stride_s, a.out_stride_h = out.stride(0), out.stride(1), out.stride(2)
        if return_lse:
            lse = torch.empty((B, H, sq), dtype=torch.float32, device=q0.device)
            a.lse = lse.data_ptr()
    if mode != _C.ATTN_FINAL:
        if acc_out is None or acc_lse is None:
            raise ValueError("acc_out and acc_lse are required for partial / merge modes")
        if acc_out.dtype != torch.float32 or acc_lse.dtype != torch.float32:
            raise TypeError("acc_out / acc_lse must be fp32")
        if tuple(acc_out.shape) != (B, sq, H, D) or not acc_out.is_contiguous():
            raise ValueError("acc_out must be contiguous (B, Sq, H, D)")
        if tuple(acc_lse.shape) != (B, H, sq) or not acc_lse.is_contiguous():
            raise ValueError("acc_lse must be contiguous (B, H, Sq)")
        a.acc_out = acc_out.data_ptr()
        a.acc_lse = acc_lse.data_ptr()
    if wait_flags is not None:
        a.n_wait = len(wait_flags.slots)
        for i, ptr in enumerate(wait_flags.slots):
            a.wait_slots[i] = ptr
        a.wait_epoch = wait_flags.epoch_ptr
        a.wait_spins = int(wait_flags.max_spins)
    a.stream = _stream_ptr(q0.device)
    n_split = 1
    if mode == _C.ATTN_FINAL:
        n_split = _pick_kv_split(q_segs, k_segs, B, H, kv_interleave) if kv_split is None else int(kv_split)
    with _on(q0.device):
        if n_split > 1:
            part_out = torch.empty((n_split, B, sq, H, D), dtype=torch.float32, device=q0.device)
            part_lse = torch.empty((n_split, B, H, sq), dtype=torch.float32, device=q0.device)
            call = lambda: _C.lib().hdit_attn_fwd_splitkv(ctypes.byref(a), n_split, part_out.data_ptr(),
                                                          part_lse.data_ptr())
        else:
            call = lambda: _C.lib().hdit_attn_fwd(ctypes.byref(a))
        if _attn_timing:
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            _C.check(call())
            e1.record()
            skv = sum(int(t.shape[1]) for t in k_segs)
            _attn_events.append((e0, e1, 4.0 * B * sq * skv * H * D))
        else:
            _C.check(call())
    _count(2 if n_split > 1 else 1)
    if not writes_out:
        return None
    if out_dsts is not None:
        return lse
    return (out, lse) if return_lse else out


_SM_COUNT = 148


def _interleave_cost(q_tiles, kv_blocks, batch, heads):
    """Cost (in KV blocks of one paired CTA) of running one query tile per CTA with the KV blocks interleaved
    over its two halves; the constants are the library's own (csrc/attn_sm100.cu)."""
    ctas_il = q_tiles * heads * batch
    return -(-ctas_il // _SM_COUNT) * ((kv_blocks + 1) // 2 * 1.12 + 6.0)


def _three_tile_cost(q_tiles, kv_lens, batch, heads):
    """The same for three query tiles per CTA over KV blocks of 96 rows (head_dim 64)."""
    ctas = -(-q_tiles // 3) * heads * batch
    return -(-ctas // _SM_COUNT) * (sum([-(-n // 96) for n in kv_lens]) + 6.0) * 1.08


def _pick_kv_split(q_segs, k_segs, batch, heads, kv_interleave=0):
    """How many ways to split the KV range. One CTA per SM runs a pair of 128-row query tiles over all KV
    blocks, so the launch takes ceil(ctas / SMs) waves; splitting the KV range s ways makes waves of 1/s the
    length and pays a fixed cost per CTA plus the merge pass. Costs are in units of one KV block of one CTA
    (about 2 us at head_dim 128), fitted to timings of 3..12 heads at 4.6k and 17.8k tokens; a split must
    promise 10 % to be taken."""
    q_lens, kv_lens = [t.shape[1] for t in q_segs], [t.shape[1] for t in k_segs]
    q_tiles = sum([(n + 127) // 128 for n in q_lens])
    ctas = (q_tiles + 1) // 2 * heads * batch
    kv_blocks = sum([(n + 127) // 128 for n in kv_lens])
    if ctas <= 0:
        return 1
    if kv_interleave == 2:
        return 1
    head_dim = q_segs[0].shape[3]
    part_bytes = batch * sum(q_lens) * heads * head_dim * 4

    def cost(s):
        waves = -(-ctas * s // _SM_COUNT)
        c = waves * (kv_blocks / s + 6.0)
        return c if s == 1 else c + 5.0 + part_bytes * s / 1e7

    best, best_cost = 1, cost(1) * 0.9
    if kv_interleave == 0 and kv_blocks >= 2:
        # without a split the library itself may interleave; a split has to beat that too
        best_cost = min(best_cost, _interleave_cost(q_tiles, kv_blocks, batch, heads) * 0.95)
    for s in (2, 3, 4):
        if kv_blocks // s >= 4 and cost(s) < best_cost:
            best, best_cost = s, cost(s)
    # or take three tiles per CTA: asked last, since most calls of a few microseconds have no split to weigh it against
    if best > 1 and head_dim == 64 and best_cost >= _three_tile_cost(q_tiles, kv_lens, batch, heads) * 0.95:
        return 1
    return best


def copy_pieces(pieces, device):
    """Moves a list of (src_ptr, dst_ptr, n_outer, src_outer_pitch, dst_outer_pitch, rows, src_pitch,
    dst_pitch, row_bytes) boxes (all byte units) on `device`'s current stream."""
    n = len(pieces)
    if n == 0:
        return
    arr = (_C.CopyPiece * n)()
    for i, pc in enumerate(pieces):
        (arr[i].src, arr[i].dst, arr[i].n_outer, arr[i].src_outer_pitch, arr[i].dst_outer_pitch, arr[i].rows,
         arr[i].src_pitch, arr[i].dst_pitch, arr[i].row_bytes) = pc
    with _on(device):
        _C.check(_C.lib().hdit_copy_pieces(arr, n, _stream_ptr(device)))
    _count((n + 39) // 40)


def copy_2d(dst, src):
    """dst[...] = src[...] for two same-shape views whose last dim is contiguous and whose leading dims
    collapse to at most (outer, rows); used for patch hand-off and slice copies."""
    if dst.shape != src.shape or dst.dtype != src.dtype:
        raise ValueError("shape / dtype mismatch")
    if dst.numel() == 0:
        return
    es = src.element_size()
    pieces = [(s.data_ptr(), d.data_ptr(), o, sop * es, dop * es, r, sp * es, dp * es, rb * es)
              for (s, d, o, sop, dop, r, sp, dp, rb) in _collapse(src, dst)]
    copy_pieces(pieces, src.device if src.is_cuda else dst.device)


def _collapse(src, dst):
    """Splits a same-shape (src, dst) view pair into 3-level boxes (element units)."""
    shape = list(src.shape)
    ss, ds = list(src.stride()), list(dst.stride())
    # drop size-1 dims, merge dims that are contiguous in both tensors
    dims = [(n, a, b) for n, a, b in zip(shape, ss, ds) if n != 1]
    if not dims:
        return [(src, dst, 1, 0, 0, 1, 0, 0, 1)]
    merged = [dims[-1]]
    for n, a, b in reversed(dims[:-1]):
        n0, a0, b0 = merged[0]
        if a == a0 * n0 and b == b0 * n0:
            merged[0] = (n * n0, a0, b0)
        else:
            merged.insert(0, (n, a, b))
    if merged[-1][1] != 1 or merged[-1][2] != 1:
        raise ValueError("innermost dimension must be contiguous in both tensors")
    row = merged[-1][0]
    lead = merged[:-1]
    if len(lead) == 0:
        return [(src, dst, 1, 0, 0, 1, 0, 0, row)]
    if len(lead) == 1:
        return [(src, dst, 1, 0, 0, lead[0][0], lead[0][1], lead[0][2], row)]
    if len(lead) == 2:
        return [(src, dst, lead[0][0], lead[0][1], lead[0][2], lead[1][0], lead[1][1], lead[1][2], row)]
    # more than two leading levels: peel the outermost
    out = []
    for i in range(shape[0]):
        out.extend(_collapse(src[i], dst[i]))
    return out


def kv_scatter(kv_cache, new_k, new_v, token_start):
    """kv_cache: (B, S, 2*R) stale buffer in the [K || V] layout; new_k / new_v: (B, n, R)-shaped views
    (any trailing dims, rows contiguous). Writes rows [token_start, token_start + n)."""
    B, S = kv_cache.shape[0], kv_cache.shape[1]
    nk = new_k.reshape(B, new_k.shape[1], -1) if new_k.dim() != 3 else new_k
    nv = new_v.reshape(B, new_v.shape[1], -1) if new_v.dim() != 3 else new_v
    n, R = nk.shape[1], nk.shape[2]
    if kv_cache.shape[2] != 2 * R or not kv_cache.is_contiguous():
        raise ValueError("kv_cache must be contiguous (B, S, 2*row)")
    if nk.stride(2) != 1 or nv.stride(2) != 1 or nk.stride() != nv.stride():
        raise ValueError("new_k / new_v rows must be contiguous and share strides")
    es = kv_cache.element_size()
    with _on(kv_cache.device):
        _C.check(_C.lib().hdit_kv_scatter(kv_cache.data_ptr(), nk.data_ptr(), nv.data_ptr(), B, S, int(token_start), n,
                                          R * es, nk.stride(1) * es, nk.stride(0) * es, _stream_ptr(kv_cache.device)))
    _count()


class FlagSignal:
    """Where an exchange kernel publishes "my rows have landed": for every peer the address (in that peer's
    memory) of the flag this rank bumps (None at this rank's own index), this rank's index, and the device
    addresses of this rank's epoch counter and ticket word."""

    def __init__(self, slots, me, epoch_ptr, ticket_ptr):
        self.slots, self.me, self.epoch_ptr, self.ticket_ptr = list(slots), int(me), int(epoch_ptr), int(ticket_ptr)


class FlagWait:
    """The matching wait: the flags in this rank's memory that the peers bump (None at this rank's own index)
    and the device address of the epoch they must reach."""

    def __init__(self, slots, epoch_ptr, max_spins=20_000_000):
        self.slots, self.epoch_ptr, self.max_spins = list(slots), int(epoch_ptr), int(max_spins)


class RawDst:
    """Destinations given as raw device addresses (e.g. mapped peer memory) plus (b, s, h) strides in elements."""

    def __init__(self, ptrs, strides):
        self.ptrs, self.strides = list(ptrs), tuple(int(x) for x in strides)

    def __len__(self):
        return len(self.ptrs)


def qk_norm_rope(tensors, *, eps=1e-6, cos=None, sin=None, rope_seq_start=0, rope_row0=0, dsts=None,
                 dst_seq_offset=0, range2=None, signal=None):
    """Fused RMSNorm + RoPE (+ head scatter) over up to three (B, S, H, D) tensors.

    tensors: list of (x, norm_weight or None, do_norm, do_rope[, norm_bias]). do_norm: False / 0 = none,
    True / 1 = RMSNorm, 2 = LayerNorm over the head dimension (weight and bias optional). dsts: None for
    in-place, or a list (one entry per tensor) of lists of destination tensors (B, S_dst, H/n_dst, D); all
    tensors share n_dst.

    range2 = (start, [(norm_weight, do_rope[, norm_bias]) per tensor], rope_row0): rows [start, S) take these norm
    weights and rotary rows instead (the norm kind stays the tensor's). signal (a FlagSignal): the kernel's last
    CTA tells the peers that this rank's rows have landed (see FlagWait / attn_fwd's wait_flags).
    """
    x0 = tensors[0][0]
    B, S, H, D = x0.shape
    a = _C.NormRopeArgs()
    a.dtype = _DTYPE_CODE[x0.dtype]
    a.batch, a.seq, a.heads, a.head_dim = B, S, H, D
    a.n_tensors = len(tensors)
    a.eps = eps
    if cos is not None:
        if cos.dtype != torch.float32 or sin.dtype != torch.float32 or not cos.is_contiguous() or not sin.is_contiguous():
            raise TypeError("cos / sin must be contiguous fp32 (rows, D) tables")
        a.cos, a.sin, a.rope_rows = cos.data_ptr(), sin.data_ptr(), cos.shape[0]
    a.rope_seq_start, a.rope_row0 = int(rope_seq_start), int(rope_row0)
    n_dst = 1 if dsts is None else len(dsts[0])
    a.n_dst = n_dst
    for i, (x, w, do_norm, do_rope, *rest) in enumerate(tensors):
        bias = rest[0] if rest else None
        if tuple(x.shape) != (B, S, H, D) or x.stride(3) != 1:
            raise ValueError("all tensors must be (B, S, H, D) with contiguous D")
        t = a.t[i]
        t.x = x.data_ptr()
        t.x_stride_b, t.x_stride_s, t.x_stride_h = x.stride(0), x.stride(1), x.stride(2)
        t.norm_weight = w.data_ptr() if w is not None else None
        t.norm_bias = bias.data_ptr() if bias is not None else None
        t.do_norm, t.do_rope = int(do_norm), int(bool(do_rope))
        outs = [x] if dsts is None else dsts[i]
        if isinstance(outs, RawDst):
            for j, ptr in enumerate(outs.ptrs):
                t.dst[j] = ptr
            t.dst_stride_b, t.dst_stride_s, t.dst_stride_h = outs.strides
        else:
            for j, o in enumerate(outs):
                t.dst[j] = o.data_ptr()
            o0 = outs[0]
            t.dst_stride_b, t.dst_stride_s, t.dst_stride_h = o0.stride(0), o0.stride(1), o0.stride(2)
        t.dst_seq_offset = int(dst_seq_offset)
    if range2 is not None:
        start, per_tensor, row0_2 = range2
        a.range2_start = int(start)
        a.range2_rope_row0 = int(row0_2)
        for i, ent in enumerate(per_tensor):
            w, do_rope, *rest = ent
            a.range2_norm_weight[i] = w.data_ptr() if w is not None else None
            a.range2_norm_bias[i] = rest[0].data_ptr() if rest and rest[0] is not None else None
            a.range2_do_rope[i] = int(bool(do_rope))
    if signal is not None:
        a.n_signal, a.signal_me = len(signal.slots), signal.me
        for i, ptr in enumerate(signal.slots):
            a.signal_slots[i] = ptr
        a.epoch_counter, a.ticket = signal.epoch_ptr, signal.ticket_ptr
    a.stream = _stream_ptr(x0.device)
    with _on(x0.device):
        _C.check(_C.lib().hdit_qk_norm_rope(ctypes.byref(a)))
    _count()


def _require_cuda(t):
    if not t.is_cuda:
        raise RuntimeError("hetu_dit_b200 kernels need CUDA tensors; there is no CPU path")


def _even_rows(x):
    return x.stride(2) == 1 and (x.shape[0] == 1 or x.stride(0) == x.shape[1] * x.stride(1))


def _rows_view(x):
    """(B, S, Dm) tensor -> (rows, dim, rows_per_batch, row_stride); rows must be evenly strided."""
    B, S, Dm = x.shape
    if not _even_rows(x):
        raise ValueError("expected a (B, S, Dm) tensor with contiguous last dim and evenly strided rows")
    return B * S, Dm, S, x.stride(1)


def ln_modulate(x, shift, scale, eps=1e-6, out=None):
    """LayerNorm(x) * (1 + scale[:, None]) + shift[:, None] for x (B, S, Dm), shift / scale (B, Dm) views."""
    _require_cuda(x)
    if out is None:
        out = torch.empty(tuple(x.shape), dtype=x.dtype, device=x.device)
    if x.shape[0] > 1 and not (_even_rows(x) and _even_rows(out)):  # e.g. a token slice of a batch: one launch per batch element
        for b in range(x.shape[0]):
            ln_modulate(x[b:b + 1], shift[b:b + 1], scale[b:b + 1], eps, out[b:b + 1])
        return out
    rows, dim, rpb, xs = _rows_view(x)
    if shift.stride(-1) != 1 or scale.stride(-1) != 1 or shift.stride(0) != scale.stride(0):
        raise ValueError("shift / scale must be (B, Dm) views with contiguous last dim and equal batch stride")
    with _on(x.device):
        _C.check(_C.lib().hdit_ln_modulate(_DTYPE_CODE[x.dtype], x.data_ptr(), shift.data_ptr(), scale.data_ptr(),
                                           out.data_ptr(), rows, dim, rpb, xs, out.stride(1), shift.stride(0), eps,
                                           _stream_ptr(x.device)))
    _count()
    return out


def ln_modulate_pair(x, x_shift, x_scale, c, c_shift, c_scale, eps=1e-6, x_out=None, c_out=None):
    """ln_modulate() of two tensors of one row length, in one launch where both are on one device and have evenly strided
    rows."""
    pair = ((x, x_shift, x_scale, x_out), (c, c_shift, c_scale, c_out))
    if not x.is_cuda or c.device != x.device or x.shape[2] != c.shape[2] or x.dtype != c.dtype or \
            not all(_even_rows(t) and (out is None or _even_rows(out)) and sh.stride(-1) == 1 and sc.stride(-1) == 1 and
                    sh.stride(0) == sc.stride(0) for t, sh, sc, out in pair):
        return ln_modulate(x, x_shift, x_scale, eps, x_out), ln_modulate(c, c_shift, c_scale, eps, c_out)
    items, outs = (_C.LnItem * 2)(), []
    for it, (t, sh, sc, out) in zip(items, pair):
        if out is None:
            out = torch.empty(tuple(t.shape), dtype=t.dtype, device=t.device)
        it.rows, dim, it.rows_per_batch, it.x_row_stride = _rows_view(t)
        it.x, it.shift, it.scale, it.out = t.data_ptr(), sh.data_ptr(), sc.data_ptr(), out.data_ptr()
        it.out_row_stride, it.mod_batch_stride = out.stride(1), sh.stride(0)
        outs.append(out)
    with _on(x.device):
        _C.check(_C.lib().hdit_ln_modulate_items(_DTYPE_CODE[x.dtype], items, 2, x.shape[2], eps, _stream_ptr(x.device)))
    _count()
    return outs


def gate_residual(x, gate, y, out=None):
    """x + gate[:, None] * y for x, y (B, S, Dm) and gate a (B, Dm) view."""
    _require_cuda(x)
    if x.shape != y.shape:
        raise ValueError("x and y differ in shape")
    if out is None:
        out = torch.empty(tuple(x.shape), dtype=x.dtype, device=x.device)
    if x.shape[0] > 1 and not (_even_rows(x) and _even_rows(y) and _even_rows(out)):
        for b in range(x.shape[0]):
            gate_residual(x[b:b + 1], gate[b:b + 1], y[b:b + 1], out[b:b + 1])
        return out
    rows, dim, rpb, xs = _rows_view(x)
    _, _, _, ys = _rows_view(y)
    with _on(x.device):
        _C.check(_C.lib().hdit_gate_residual(_DTYPE_CODE[x.dtype], x.data_ptr(), gate.data_ptr(), y.data_ptr(),
                                             out.data_ptr(), rows, dim, rpb, xs, ys, out.stride(1), gate.stride(0),
                                             _stream_ptr(x.device)))
    _count()
    return out


def gelu_tanh(x, out=None):
    """tanh-approximated GELU over the last dim of a (B, S, Dm) tensor with evenly strided rows; `out` may be
    `x` itself or a column block of a wider buffer with the same (B, S)."""
    _require_cuda(x)
    rows, dim, _, xs = _rows_view(x)
    if out is None:
        out = torch.empty(tuple(x.shape), dtype=x.dtype, device=x.device)
    rows_o, dim_o, _, os_ = _rows_view(out)
    if (rows_o, dim_o) != (rows, dim):
        raise ValueError("out differs from x in shape")
    with _on(x.device):
        _C.check(_C.lib().hdit_gelu_tanh(_DTYPE_CODE[x.dtype], x.data_ptr(), out.data_ptr(), rows, dim, xs, os_,
                                         _stream_ptr(x.device)))
    _count()
    return out


def linear_fused(x, weight, bias=None, epilogue="bias", residual=None, gate=None, out=None, tile_n=0, max_ctas=0,
                 tile_m=0, cta_pair=0):
    """epilogue(x @ weight.T + bias) in one tensor-core kernel (csrc/gemm_sm100.cu). x (B, S, K) or (rows, K) with
    evenly strided rows, weight (N, K) as torch.nn.Linear stores it. epilogue: "bias" (a plain linear layer),
    "gelu_tanh", or "gate_residual" = residual + gate[:, None, :] * linear(x) with gate (B, N) and residual of the
    output's shape. `out` may be a column block of a wider buffer, or `residual` itself."""
    _require_cuda(x)
    if x.dim() == 2:
        res3 = residual.unsqueeze(0) if residual is not None else None
        out3 = out.unsqueeze(0) if out is not None else None
        return linear_fused(x.unsqueeze(0), weight, bias, epilogue, res3, gate, out3, tile_n, max_ctas, tile_m, cta_pair)[0]
    rows, k, _, xs = _rows_view(x)
    n = weight.shape[0]
    if weight.dim() != 2 or weight.shape[1] != k or weight.stride(1) != 1 or weight.dtype != x.dtype:
        raise ValueError("weight must be (N, K), K-contiguous, of x's dtype")
    if out is None:
        out = torch.empty(tuple(x.shape[:-1]) + (n,), dtype=x.dtype, device=x.device)
    rows_o, n_o, _, os_ = _rows_view(out)
    if (rows_o, n_o) != (rows, n) or out.dtype != x.dtype:
        raise ValueError("out does not match (rows, N) or x's dtype")
    a = _C.GemmArgs()
    a.dtype = _DTYPE_CODE[x.dtype]
    a.epilogue = {"bias": _C.GEMM_BIAS, "gelu_tanh": _C.GEMM_BIAS_GELU_TANH,
                  "gate_residual": _C.GEMM_BIAS_GATE_RESIDUAL}[epilogue]
    a.m, a.n, a.k = rows, n, k
    a.a, a.lda = x.data_ptr(), xs
    a.w, a.ldw = weight.data_ptr(), weight.stride(0)
    if bias is not None:
        if bias.numel() != n or not bias.is_contiguous() or bias.dtype != x.dtype:
            raise ValueError("bias must be N contiguous elements of x's dtype")
        a.bias = bias.data_ptr()
    a.out, a.ldo = out.data_ptr(), os_
    if epilogue == "gate_residual":
        rows_r, n_r, _, rs = _rows_view(residual)
        if (rows_r, n_r) != (rows, n) or residual.dtype != x.dtype:
            raise ValueError("residual does not match (rows, N) or x's dtype")
        if gate.dim() != 2 or gate.shape[1] != n or gate.stride(1) != 1 or rows % gate.shape[0] != 0 or gate.dtype != x.dtype:
            raise ValueError("gate must be (B, N) of x's dtype with rows a multiple of B")
        a.residual, a.ldr = residual.data_ptr(), rs
        a.gate, a.gate_batch_stride = gate.data_ptr(), gate.stride(0)
        a.rows_per_batch = rows // gate.shape[0]
    a.tile_n, a.max_ctas, a.tile_m, a.cta_pair = tile_n, max_ctas, tile_m, cta_pair
    with _on(x.device):
        a.stream = _stream_ptr(x.device)
        _C.check(_C.lib().hdit_linear_fused(ctypes.byref(a)))
    _count()
    return out


class Lin:
    """One linear layer of a linear_group() call: y = tail(x @ weight.T + bias). x (B, S, K) with evenly strided rows.

    epilogue "bias", "gelu_tanh", "gate_residual" (residual, gate) as in linear_fused(), or "norm_rope": per-head norm
    (norm = (kind, weight, bias, eps), kind 1 RMSNorm, 2 LayerNorm with head_dim 64, None for no norm) and rotary
    embedding (rope = (rope_seq_start, rope_row0) into the call's cos / sin tables, None for no rotation) over heads of
    `head_dim` columns, as qk_norm_rope() computes them."""
    __slots__ = ("x", "weight", "bias", "epilogue", "residual", "gate", "out", "head_dim", "norm", "rope")

    def __init__(self, x, linear, epilogue="bias", residual=None, gate=None, out=None, head_dim=0, norm=None, rope=None):
        self.x, self.weight, self.bias, self.epilogue = x, linear.weight, linear.bias, epilogue
        self.residual, self.gate, self.out = residual, gate, out
        self.head_dim, self.norm, self.rope = head_dim, norm, rope

    def _even(self):
        return self.x.shape[0] == 1 or all(t is None or _even_rows(t) for t in (self.x, self.residual, self.out))

    def _entry(self, b):
        """This layer on one batch entry."""
        e = Lin.__new__(Lin)
        for name in self.__slots__:
            v = getattr(self, name)
            setattr(e, name, v[b:b + 1] if name in ("x", "residual", "gate", "out") and v is not None else v)
        return e

    def _entries(self):
        """[self], or one layer per batch entry where rows are not evenly strided over the batch (a slice of the rows of
        every entry)."""
        if self._even():
            return [self]
        if self.out is None:
            self.out = torch.empty((self.x.shape[0], self.x.shape[1], self.weight.shape[0]), dtype=self.x.dtype,
                                   device=self.x.device)
        return [self._entry(b) for b in range(self.x.shape[0])]


_EPILOGUES = {"bias": _C.GEMM_BIAS, "gelu_tanh": _C.GEMM_BIAS_GELU_TANH, "gate_residual": _C.GEMM_BIAS_GATE_RESIDUAL,
              "norm_rope": _C.GEMM_BIAS_NORM_ROPE}


def linear_group(items, cos=None, sin=None, tile_m=0, tile_n=0, cta_pair=0, max_ctas=0):
    """Several independent linear layers with one inner dimension in one launch (csrc/gemm_sm100.cu), see Lin. A layer
    whose rows are not evenly strided over the batch counts once per batch entry. No item may read what another one
    writes. Returns their results in order."""
    x0 = items[0].x
    _require_cuda(x0)
    whole, items = items, [e for it in items for e in it._entries()]
    if not 1 <= len(items) <= _C.MAX_LINEAR_ITEMS:
        raise ValueError("between 1 and %d linear layers" % _C.MAX_LINEAR_ITEMS)
    a = _C.LinearGroupArgs()
    a.dtype, a.n_items, a.k = _DTYPE_CODE[x0.dtype], len(items), x0.shape[2]
    a.tile_m, a.tile_n, a.cta_pair, a.max_ctas = tile_m, tile_n, cta_pair, max_ctas
    if cos is not None:
        if cos.dtype != torch.float32 or sin.dtype != torch.float32 or not cos.is_contiguous() or not sin.is_contiguous() \
                or cos.shape != sin.shape:
            raise TypeError("cos / sin must be contiguous fp32 (rows, D) tables")
        a.cos, a.sin, a.rope_rows = cos.data_ptr(), sin.data_ptr(), cos.shape[0]
    x_prev = None
    for it, d in zip(items, a.item):
        x, w, bias, out = it.x, it.weight, it.bias, it.out
        if x is not x_prev:
            rows, k, rpb, xs = _rows_view(x)
            x_prev, x_ptr = x, x.data_ptr()
        n = w.shape[0]
        if w.dim() != 2 or w.shape[1] != k or k != a.k or w.stride(1) != 1 or w.dtype != x0.dtype or x.dtype != x0.dtype:
            raise ValueError("every weight must be (N, K), K-contiguous, of x's dtype, with one K")
        if out is None:
            out = it.out = torch.empty((x.shape[0], x.shape[1], n), dtype=x.dtype, device=x.device)
        rows_o, n_o, _, os_ = _rows_view(out)
        if (rows_o, n_o) != (rows, n) or out.dtype != x.dtype:
            raise ValueError("out does not match (rows, N)")
        d.m, d.n, d.a, d.lda, d.w, d.ldw = rows, n, x_ptr, xs, w.data_ptr(), w.stride(0)
        if bias is not None:
            if bias.numel() != n or not bias.is_contiguous() or bias.dtype != x.dtype:
                raise ValueError("bias must be N contiguous elements of x's dtype")
            d.bias = bias.data_ptr()
        d.out, d.ldo, d.epilogue, d.rows_per_batch = out.data_ptr(), os_, _EPILOGUES[it.epilogue], rpb
        if it.epilogue == "gate_residual":
            rows_r, n_r, _, rs = _rows_view(it.residual)
            if (rows_r, n_r) != (rows, n) or it.residual.dtype != x.dtype:
                raise ValueError("residual does not match (rows, N)")
            gate = it.gate
            if gate.dim() != 2 or tuple(gate.shape) != (x.shape[0], n) or gate.stride(1) != 1 or gate.dtype != x.dtype:
                raise ValueError("gate must be (B, N)")
            d.residual, d.ldr, d.gate, d.gate_batch_stride = it.residual.data_ptr(), rs, gate.data_ptr(), gate.stride(0)
        elif it.epilogue == "norm_rope":
            d.head_dim = it.head_dim
            if it.norm is not None:
                d.norm, nw, nb, d.eps = it.norm
                for t in (nw, nb):
                    if t is not None and (t.dtype != x.dtype or t.numel() != it.head_dim or not t.is_contiguous()):
                        raise ValueError("norm weight / bias must be head_dim contiguous elements of x's dtype")
                d.norm_weight = nw.data_ptr() if nw is not None else None
                d.norm_bias = nb.data_ptr() if nb is not None else None
            if it.rope is not None:
                if cos is None or cos.shape[1] != it.head_dim:
                    raise ValueError("rope needs cos / sin tables of head_dim columns")
                d.rope, d.rope_seq_start, d.rope_row0 = 1, int(it.rope[0]), int(it.rope[1])
    with _on(x0.device):
        a.stream = _stream_ptr(x0.device)
        _C.check(_C.lib().hdit_linear_group(ctypes.byref(a)))
    _count()
    return [it.out for it in whole]


# Whether linear layers may run the fused tensor-core kernel (csrc/gemm_sm100.cu) instead of the library GEMM followed by
# one-pass kernels, for which tails, and from / to how many rows (an input's rows count once, however many layers of a
# launch read it) on top of the rule in _group_pays(). HDIT_FUSED_LINEAR=0 turns the fused kernel off,
# HDIT_FUSED_LINEAR_TAILS=gelu_tanh fuses only that tail; "bias" and "norm_rope" are the Q, K, V projections.
FUSED_LINEAR = os.environ.get("HDIT_FUSED_LINEAR", "1") == "1"
FUSED_LINEAR_TAILS = set(os.environ.get("HDIT_FUSED_LINEAR_TAILS", "bias,gelu_tanh,gate_residual,norm_rope").split(","))
FUSED_LINEAR_MIN_ROWS = int(os.environ.get("HDIT_FUSED_LINEAR_MIN_ROWS", "0"))
FUSED_LINEAR_MAX_ROWS = int(os.environ.get("HDIT_FUSED_LINEAR_MAX_ROWS", str(1 << 40)))


_HOOKS_OF_ALL, _PRE_HOOKS_OF_ALL = _all_modules._global_forward_hooks, _all_modules._global_forward_pre_hooks


def is_plain(module, cls):
    """Whether calling `module` runs cls.forward and nothing else, so that what it does may be done without the call: no
    other class (an adapter, a quantised layer), no forward() put on the object, and no hook, of this module or of all
    modules, that waits for the call."""
    if type(module) is not cls:
        return False
    own = module.__dict__  # what a module's attributes are read from, at a quarter of the cost
    return not (own["_forward_hooks"] or own["_forward_pre_hooks"] or "forward" in own or _HOOKS_OF_ALL or _PRE_HOOKS_OF_ALL)


def _plain_weights(linear):
    """(weight, bias) where calling `linear` is x @ weight.T + bias and nothing else, so that a kernel may be given them
    instead: a plain torch.nn.Linear without a weight of a tensor class of its own. Else None."""
    if not is_plain(linear, torch.nn.Linear):
        return None
    own = linear.__dict__["_parameters"]
    w, b = own.get("weight"), own.get("bias")
    if type(w) is not torch.nn.Parameter or (linear.bias is not None if b is None else type(b) is not torch.nn.Parameter):
        return None
    return w, b


def linear_tail(linear, x, epilogue, residual=None, gate=None, out=None):
    """A torch.nn.Linear followed by its elementwise tail ("gelu_tanh", or "gate_residual" = residual +
    gate[:, None] * linear(x)), as one kernel when _fusable_weights() has the layer, rows are evenly strided across
    the batch and it pays, else as the call of `linear` plus hdit_gelu_tanh / hdit_gate_residual."""
    if epilogue not in ("gelu_tanh", "gate_residual"):
        raise ValueError(epilogue)
    weights = _fusable_weights((x,), (linear,)) if epilogue in FUSED_LINEAR_TAILS else None
    if weights is not None:
        (w, b), = weights
        (B, S, k), n = x.shape, w.shape[0]
        if _even_rows(x) and FUSED_LINEAR_MIN_ROWS <= B * S <= FUSED_LINEAR_MAX_ROWS and _tail_fits(x, n, residual, gate, out) \
                and (residual is None or _even_rows(residual)) and (out is None or _even_rows(out)) and _group_pays(((B * S, n),), k):
            return linear_fused(x, w, b, epilogue, residual=residual, gate=gate, out=out)
    y = linear(x)
    if epilogue == "gelu_tanh":
        return gelu_tanh(y, out=y if out is None else out)
    return gate_residual(residual, gate, y, out=out)


def _aligned(x):
    """Whether the rows of a (B, S, Dm) tensor are contiguous, do not overlap and start on 16-byte boundaries (16-bit
    elements)."""
    (B, _, dim), (sb, ss, sk) = x.shape, x.stride()
    return sk == 1 and ss >= dim and ss % 8 == 0 and (B == 1 or sb % 8 == 0) and x.data_ptr() % 16 == 0


def _tail_fits(x, n, residual, gate, out=None):
    """Whether the kernel takes these with an (B, S, N) output for input x: residual and result of that shape and gate
    (B, N), of x's type, on its device, aligned. What it does not take, gate_residual() takes or refuses by itself."""
    B, S, _ = x.shape
    dtype, dev = x.dtype, x.device
    for t in (residual, out):
        if t is not None and (t.shape != (B, S, n) or t.dtype != dtype or t.device != dev or not _aligned(t)):
            return False
    if gate is None:
        return True
    return gate.shape == (B, n) and gate.dtype == dtype and gate.device == dev and gate.stride(1) == 1 and \
        gate.stride(0) % 8 == 0 and gate.data_ptr() % 16 == 0


def _fusable_weights(xs, linears):
    """The (weight, bias) of every layer where these layers on these (B, S, K) inputs may go through linear_fused() /
    linear_group(): the switch is on, no gradient is recorded, the layers are plain torch.nn.Linear that nothing waits for
    the call of, and layouts and types are what the kernel takes. Else None: the library GEMM takes inner sizes that are no
    multiple of 8 and rows that overlap or do not start on 16-byte boundaries."""
    if not FUSED_LINEAR or torch.is_grad_enabled():
        return None
    k, dtype, dev = xs[0].shape[-1], xs[0].dtype, xs[0].device
    if dtype not in _DTYPE_CODE or k % 8:
        return None
    for x in xs:
        if not x.is_cuda or x.dim() != 3 or x.dtype != dtype or x.device != dev:
            return None
        B, S, kx = x.shape
        if kx != k or (B > 1 and S < 32) or not _aligned(x):
            return None
    weights = []
    for linear in linears:
        plain = _plain_weights(linear)
        if plain is None:
            return None
        w, b = plain
        (n, kw), (sn, sk) = w.shape, w.stride()
        if kw != k or n % 8 or sk != 1 or sn < k or sn % 8 or w.dtype != dtype or w.device != dev or w.data_ptr() % 16:
            return None
        if b is not None and (b.dtype != dtype or b.numel() != n or not b.is_contiguous() or b.data_ptr() % 16):
            return None
        weights.append(plain)
    return weights


def can_group_linears(xs, linears):
    """Whether these layers on these inputs may go through linear_group(), see _fusable_weights()."""
    return _fusable_weights(xs, linears) is not None


def norm_rope_fits(x, head_dim, norms, rope):
    """Whether the "norm_rope" epilogue of linear_group() takes these norms, (kind, weight, bias, eps) each, and rotary
    tables (cos, sin) or None for input x. qk_norm_rope() takes more: LayerNorm of 128-wide heads, for which the epilogue
    has no registers left, and tables of different lengths."""
    if head_dim not in (64, 128):
        return False
    for kind, w, b, _ in norms:
        if kind not in (1, 2) or (kind == 2 and head_dim != 64):
            return False
        for t in (w, b):
            if t is not None and (t.dtype != x.dtype or t.device != x.device or t.numel() != head_dim or
                                  not t.is_contiguous() or t.data_ptr() % 16):
                return False
    return rope is None or (rope[0].shape == rope[1].shape and rope[0].dim() == 2 and rope[0].shape[1] == head_dim and
                            all(t.dtype == torch.float32 and t.is_contiguous() and t.data_ptr() % 16 == 0 for t in rope))


_WIDE_TILES = ((128, 256, _SM_COUNT, 2.36), (128, 128, _SM_COUNT, 1.25), (256, 256, _SM_COUNT // 2, 2.1))
_TILES_WIDE_HEADS = _WIDE_TILES + ((256, 128, _SM_COUNT // 2, 1.2),)  # 192 columns do not hold whole heads of 128
_TILES = _TILES_WIDE_HEADS + ((256, 192, _SM_COUNT // 2, 1.725),)


def _group_cost(shapes, tile_shapes=_TILES):
    """Time of one launch over the (rows, n, ...) output shapes in units of one SM's work on a 128 x 128 block of output:
    waves of output tiles times the time of a tile, smallest over the tile shapes (rows, columns, how many at a time, time;
    the library's own, csrc/gemm_sm100.cu). Second result: the same if every SM always had work."""
    best = None
    for tm, tn, units, per_tile in tile_shapes:
        tiles = sum(-(-m // tm) * -(-n // tn) for m, n, *_ in shapes)
        cost = -(-tiles // units) * per_tile
        best = cost if best is None else min(best, cost)
    return best, sum(m * n for m, n, *_ in shapes) / 16384.0 / _SM_COUNT


# An SM takes 4 cycles per unit of the inner dimension for a 128 x 128 block: 2.3 ns. What a separate library GEMM plus
# tail kernel costs beyond its arithmetic, and how far the library is from the kernel's best rate.
_NS_PER_K, _SAVED_US_PER_LAYER, _LIBRARY_RATE = 2.3e-3, 5.0, 1.15


@functools.lru_cache(maxsize=4096)
def _group_pays(shapes, k):
    """Whether one launch over these outputs, (rows, n) each or (rows, n, 128) with a norm + rotation tail over heads of
    128, beats a library GEMM and a tail kernel per layer: what the partly filled last wave wastes (the library splits K
    there) has to stay below what the launches and the extra pass over the output cost. Measured in bursts of 20 ms, us,
    this kernel / library: 2 layers of 1961 + 231 rows, K = 12288: 127 / 132 (192-column tiles); K = 3072: 36 / 44; 1024 +
    256 rows, K = 12288: 83 / 93; 256 + 77 rows, K = 12288: 45 / 45 (not taken); 4096 + 512 rows, K = 12288: 253 / 274;
    12240 + 224 rows: 671 / 660 (taken although 2 % slower alone); Q, K, V of 2 x (1024 + 77) rows, K = 1536: 27 / 41, of
    4096 + 512 rows, K = 3072 with norm and rotation: 193 / 252.

    The narrow tiles of a pair count for several layers only: for one the library has narrow tiles and split K as well.
    One layer that they alone would bring here, kernel / library, us in bursts | in loops at the power limit: 2290 rows,
    K = 15360, N = 3072: 150 / 141 | 179 / 169; K = 12288: 124 / 117 | 146 / 139; 2265 rows, K = 6144, N = 1536: 35 / 34;
    498 rows, K = 3072, N = 12288: 37 / 35. One layer that 256-column tiles bring here is about even: K = 15360, N = 3072,
    2816 rows 183 / 180 | 217 / 209; 4352: 272 / 276 | 324 / 326; 5696: 368 / 383 | 435 / 426; 7456: 480 / 489 | 556 / 566;
    8900: 563 / 554 | 661 / 645; 14656: 925 / 924 | 1091 / 1060; 16896: 1025 / 1082 | 1236 / 1236."""
    wide_heads = any([len(s) == 3 for s in shapes])
    cost, ideal = _group_cost(shapes, _WIDE_TILES if len(shapes) == 1 else _TILES_WIDE_HEADS if wide_heads else _TILES)
    return (cost - _LIBRARY_RATE * ideal) * k * _NS_PER_K <= _SAVED_US_PER_LAYER * len(shapes)


def use_linear_group(items):
    """Whether one linear_group() launch beats separate library GEMMs and tail kernels."""
    shapes, inputs = [], {}
    for it in items:
        if it.epilogue not in FUSED_LINEAR_TAILS:
            return False
        B, S, k = it.x.shape
        n = it.weight.shape[0]
        tail = (128,) if it.epilogue == "norm_rope" and it.head_dim == 128 else ()
        shapes += [(B * S, n, *tail)] if it._even() else [(S, n, *tail)] * B
        inputs[id(it.x)] = B * S
    return 1 <= len(shapes) <= _C.MAX_LINEAR_ITEMS and \
        FUSED_LINEAR_MIN_ROWS <= sum(inputs.values()) <= FUSED_LINEAR_MAX_ROWS and _group_pays(tuple(shapes), k)


def try_linear_tails(specs):
    """The layers of linear_tails() in one launch, or None where that is not possible or does not pay."""
    weights = _fusable_weights([sp[1] for sp in specs], [sp[0] for sp in specs])
    if weights is None:
        return None
    items = []
    for (linear, x, epilogue, *rest), (w, _) in zip(specs, weights):
        residual, gate = rest if rest else (None, None)
        if not _tail_fits(x, w.shape[0], residual, gate):
            return None
        items.append(Lin(x, linear, epilogue, residual=residual, gate=gate))
    return linear_group(items) if use_linear_group(items) else None


def linear_tails(specs):
    """linear_tail() of several independent layers, specs = [(linear, x, epilogue[, residual, gate])]: in one launch where
    that is possible and pays, else one after the other."""
    outs = try_linear_tails(specs)
    if outs is None:
        outs = [linear_tail(l, x, ep, residual=rest[0] if rest else None, gate=rest[1] if rest else None)
                for l, x, ep, *rest in specs]
    return outs


def cfg_euler_step(noise_pred, sample, sigmas, step_index, guidance_scale, cfg=True, out=None, out_peer_ptr=None):
    """sample + (sigmas[i + 1] - sigmas[i]) * guided(noise_pred) in one pass. noise_pred is (2 * B, ...) =
    [unconditional; conditional] when cfg is set (guided = uncond + scale * (cond - uncond)), else (B, ...) taken as
    it is; sample and the result are (B, ...), contiguous, 16-bit. sigmas: fp32 device tensor. out_peer_ptr: raw
    device address (e.g. the next pipeline stage's inbox slot) that receives a second copy of the result."""
    _require_cuda(sample)
    if not (noise_pred.is_contiguous() and sample.is_contiguous()):
        raise ValueError("noise_pred and sample must be contiguous")
    n = sample.numel()
    if noise_pred.numel() != (2 * n if cfg else n):
        raise ValueError("noise_pred does not match sample")
    if sigmas.dtype != torch.float32 or not sigmas.is_cuda or not 0 <= step_index < sigmas.numel() - 1:
        raise ValueError("sigmas must be a float32 device tensor with step_index + 1 in range")
    if out is None:
        out = torch.empty_like(sample)
    es = noise_pred.element_size()
    uncond = noise_pred.data_ptr()
    cond = uncond + n * es if cfg else None
    with _on(sample.device):
        _C.check(_C.lib().hdit_cfg_euler_step(_DTYPE_CODE[sample.dtype], uncond, cond, sample.data_ptr(), out.data_ptr(),
                                              out_peer_ptr, n, float(guidance_scale), sigmas.data_ptr(), int(step_index),
                                              _stream_ptr(sample.device)))
    _count()
    return out
