"""Host glue between torch tensors and the C ABI (ft_decode / ft_stage1 / ft_stage2).

Mirrors the call contract of the reference's ``fasttree_decode``
(kernel_bench/fasttree.py:582-642): the caller owns every tensor, kernels are
enqueued on torch's current CUDA stream, nothing synchronises with the host and
nothing is allocated per call.  Bad arguments raise ``FastTreeError`` /
``ValueError`` instead of silently producing garbage.
"""
import ctypes
import weakref

import torch

from . import lib as _lib

# What is remembered about a plan: per vnode_to_q_entries table (by tensor object, weakly) whether it carries row ranges
# (:func:`split_q_entries`).  id(tensor) -> (weak reference to it, (version, data_ptr, numel), rows or -1)
_RANGE_CACHE = {}


def _require_cuda(name, t):
    if not isinstance(t, torch.Tensor):
        raise ValueError(f"{name} must be a torch.Tensor")
    if not t.is_cuda:
        raise ValueError(f"{name} is on {t.device}; the engine has no CPU path - tensors must live on a CUDA device")


def _table(name, t):
    _require_cuda(name, t)
    if t.dtype != torch.int32:
        raise ValueError(f"{name} must be int32, got {t.dtype}")
    if not t.is_contiguous():
        raise ValueError(f"{name} must be contiguous")
    return t


ROW_RANGE_MAGIC = 0x46545252          # "FTRR": trailer of a vnode_to_q_entries table that carries row ranges


def _version_of(t):
    """In-place-write counter of a tensor; tensors created under ``torch.inference_mode()`` keep none (a serving
    host runs its decode loop there), and for those the answer is a constant."""
    try:
        return t._version
    except RuntimeError:
        return -1


def pack_row_ranges(q_entries, ranges):
    """The B200 plan format's optional tenth table - per partial row the tokens
    ``[begin, end)`` of its vnode's KV chunk that the row attends to (int32
    ``[rows, 2]``) - has no slot in the reference's 13-entry tuple.  It travels
    INSIDE the ``vnode_to_q_entries`` table it is parallel to:

        [ R request ids | 2R range entries | ROW_RANGE_MAGIC, R ]

    so that clone(), .to(), .contiguous(), pickling or rebuilding the tuple keep it.
    Takes and returns numpy int32 arrays."""
    import numpy as np
    rows = int(q_entries.shape[0])
    if ranges.shape != (rows, 2):
        raise ValueError("the row-range table needs two entries per partial row")
    tail = np.array([ROW_RANGE_MAGIC, rows], dtype=np.int32)
    return np.ascontiguousarray(np.concatenate([q_entries.astype(np.int32), ranges.astype(np.int32).ravel(), tail]))


def split_q_entries(vnode_to_q_entries):
    """``(rows, ranges)`` of a vnode_to_q_entries table: the number of partial rows it
    names and a ``[rows, 2]`` view of the row ranges packed behind them (None for
    a table in the reference's format).  Recognising the trailer reads two
    integers back from the device; the answer is remembered per tensor object
    (weakly, and re-read when the tensor was written to in place or re-allocated), so
    a steady decode loop does not repeat it.
    The first call on a new table therefore synchronises with the device and
    must not fall inside a CUDA graph capture."""
    t = vnode_to_q_entries
    n = t.numel()
    if n < 5 or (n - 2) % 3 != 0:                 # too short for a trailer, or no multiple of three entries before it
        return n, None
    state = (_version_of(t), t.data_ptr(), n)
    ident = id(t)
    known = _RANGE_CACHE.get(ident)
    if known is not None and known[0]() is t and known[1] == state:
        hit = known[2]
    else:
        magic, rows = t.view(-1)[-2:].tolist()
        hit = rows if magic == ROW_RANGE_MAGIC and 3 * rows + 2 == n else -1
        _RANGE_CACHE[ident] = (weakref.ref(t, lambda _r, k=ident: _RANGE_CACHE.pop(k, None)), state, hit)
    if hit < 0:
        return n, None
    return hit, t.view(-1)[hit:3 * hit].view(hit, 2)


def row_ranges_of(vnode_to_q_entries):
    return split_q_entries(vnode_to_q_entries)[1]


_ARG_NAMES = ("q", "k_buffer", "v_buffer", "o", "vnode_to_kv_entries", "vnode_to_kv_offs", "vnode_to_kv_lens",
              "vnode_to_q_entries", "vnode_to_q_offs", "vnode_to_q_lens", "req_to_vnode_entries", "req_to_vnode_offs",
              "req_to_vnode_lens", "mid_o", "mid_lse", "phase_node_nums", "phase_node_offsets", "phase_q_tile_sizes",
              "phase_kv_tile_sizes", "sm_scale")


def _resolve(args, path, row_ranges):
    """``(path code, row-range tensor or None, partial rows or -1)`` of a call's arguments."""
    if len(args) != len(_ARG_NAMES):
        raise TypeError(f"expected {len(_ARG_NAMES)} positional arguments, got {len(args)}")
    code = _lib.PATHS.get(path)
    if code is None:
        raise ValueError(f"path must be one of {sorted(_lib.PATHS)}")
    if isinstance(row_ranges, str):
        if row_ranges != "detect":
            raise ValueError("row_ranges must be 'detect', None or an int32 tensor")
        _table("vnode_to_q_entries", args[7])
        rows, ranges = split_q_entries(args[7])
        return code, ranges, rows
    return code, row_ranges, -1


def build_args(*args, path="auto", o_lse=None, stream=None, row_ranges="detect", phase_info=None, kv_entries_aux=None,
               logit_cap=-1, **named):
    """A filled :class:`DecodeArgs` struct; raises ``ValueError`` where a tensor does not fit.  Positional arguments
    are those of the reference's ``fasttree_decode`` up to and including ``sm_scale`` (and ``logit_cap``); they may also
    be given by name.
    ``kv_entries_aux``: an int32 CUDA tensor, the second row-id table that vnodes with bit 30 of their
    ``vnode_to_kv_offs`` value set read (grouped private tails of the serving path).  ``phase_info``: an
    int32 CUDA tensor ``[n0, n1, o0, o1]`` that stage 1 reads on the device in
    place of ``phase_node_nums`` / ``phase_node_offsets`` (the launch then does not
    depend on the plan and survives a re-plan inside a captured CUDA graph).  ``row_ranges``:
    ``"detect"`` looks for ranges packed into ``vnode_to_q_entries`` (see
    :func:`pack_row_ranges`), ``None`` says the plan has none (no look-up, no
    device read), a tensor gives the table explicitly."""
    if len(args) == len(_ARG_NAMES) + 1:
        args, logit_cap = args[:-1], args[-1]
    if named:
        missing = [n for n in _ARG_NAMES[len(args):] if n not in named]
        if missing or len(named) != len(_ARG_NAMES) - len(args):
            raise TypeError(f"build_args: missing {missing}, unknown or repeated {sorted(set(named) - set(_ARG_NAMES[len(args):]))}")
        args = args + tuple(named[n] for n in _ARG_NAMES[len(args):])
    code, ranges, rows = _resolve(args, path, row_ranges)
    raw = _lib.call_module().args(args, logit_cap, code, o_lse, ranges, rows, phase_info, kv_entries_aux,
                                  -1 if stream is None else stream)
    return _lib.DecodeArgs.from_buffer_copy(raw)


_ENTRIES = {"ft_decode": 0, "ft_stage1": 1, "ft_stage2": 2}


def _call(fn_name, args, logit_cap, path, o_lse, row_ranges, phase_info=None, kv_entries_aux=None):
    code, ranges, rows = _resolve(args, path, row_ranges)
    rc = _lib.call_module().call(_ENTRIES[fn_name], args, logit_cap, code, o_lse, ranges, rows, phase_info, kv_entries_aux, -1)
    if rc != 0:
        _lib.check(rc)


def decode(*args, logit_cap=-1, path="auto", o_lse=None, row_ranges="detect", phase_info=None, kv_entries_aux=None):
    """Stage 1 + stage 2.  Positional arguments are those of the reference's
    ``fasttree_decode`` up to and including ``sm_scale``."""
    _call("ft_decode", args, logit_cap, path, o_lse, row_ranges, phase_info, kv_entries_aux)


def stage1(*args, logit_cap=-1, path="auto", row_ranges="detect", phase_info=None, kv_entries_aux=None):
    _call("ft_stage1", args, logit_cap, path, None, row_ranges, phase_info, kv_entries_aux)


def stage2(*args, logit_cap=-1, o_lse=None):
    _call("ft_stage2", args, logit_cap, "auto", o_lse, None)


def decode_host_io(q_host, o_host, q_dev, k_buffer, v_buffer, o_dev, *rest, logit_cap=-1, path="auto",
                   row_ranges="detect", wait=True):
    """One decode step fed from and drained to pinned host memory through ONE C-ABI call
    (``ft_decode_host_io``): ``q_host`` -> ``q_dev`` (one cudaMemcpyAsync), stage 1 + stage 2, ``o_dev`` ->
    ``o_host`` (one cudaMemcpyAsync), all on torch's current stream; ``wait`` synchronises that stream before
    returning, so ``o_host`` is valid.  ``q_dev`` / ``o_dev`` are caller-owned packed device staging tensors,
    ``rest`` are the plan tables, scratch, phase lists, tile lists and ``sm_scale`` as in :func:`decode`."""
    for name, t in (("q_host", q_host), ("o_host", o_host)):
        if not isinstance(t, torch.Tensor) or t.is_cuda or not t.is_pinned() or not t.is_contiguous():
            raise ValueError(f"{name} must be a contiguous pinned host tensor")
    if q_host.shape != q_dev.shape or o_host.shape != o_dev.shape or q_host.dtype != q_dev.dtype \
            or o_host.dtype != o_dev.dtype:
        raise ValueError("host and device staging tensors must agree in shape and dtype")
    if not q_dev.is_contiguous() or not o_dev.is_contiguous():
        raise ValueError("the device staging tensors must be packed")
    tensors = (q_dev, k_buffer, v_buffer, o_dev) + tuple(rest[:11])
    pn, po, pq, pk, sm_scale = rest[11:16]
    a = build_args(*tensors, pn, po, pq, pk, sm_scale, logit_cap, path=path, row_ranges=row_ranges)
    lib = _lib.load()
    if q_dev.device.index != torch.cuda.current_device():
        with torch.cuda.device(q_dev.device):
            rc = lib.ft_decode_host_io(ctypes.byref(a), q_host.data_ptr(), o_host.data_ptr(), 1 if wait else 0)
    else:
        rc = lib.ft_decode_host_io(ctypes.byref(a), q_host.data_ptr(), o_host.data_ptr(), 1 if wait else 0)
    _lib.check(rc)


def prepare_host_io(q_host, o_host, q_dev, k_buffer, v_buffer, o_dev, *rest, logit_cap=-1, path="auto",
                    row_ranges="detect", wait=True):
    """A prepared :func:`decode_host_io`: validates once, fills the argument block once and returns a callable
    whose only work is the foreign call (on the CUDA stream that is current when it is CALLED).  The callable
    keeps every tensor alive; build a new one when a tensor is replaced."""
    decode_host_io(q_host, o_host, q_dev, k_buffer, v_buffer, o_dev, *rest, logit_cap=logit_cap, path=path,
                   row_ranges=row_ranges, wait=True)          # validation, first-use costs, range look-up
    pn, po, pq, pk, sm_scale = rest[11:16]
    tensors = (q_dev, k_buffer, v_buffer, o_dev) + tuple(rest[:11])
    a = build_args(*tensors, pn, po, pq, pk, sm_scale, logit_cap, path=path, row_ranges=row_ranges)
    fn = _lib.load().ft_decode_host_io
    ref, qp, op, flag = ctypes.byref(a), q_host.data_ptr(), o_host.data_ptr(), 1 if wait else 0
    keep = (tensors, q_host, o_host, a)
    device = q_dev.device

    def run(_keep=keep):
        a.stream = torch.cuda.current_stream(device).cuda_stream
        rc = fn(ref, qp, op, flag)
        if rc != 0:
            _lib.check(rc)

    return run


def stage1_path_name(*args, logit_cap=-1, path="auto"):
    a = build_args(*args, logit_cap, path=path)
    name = _lib.load().ft_stage1_path_name(ctypes.byref(a))
    if name is None:
        _lib.check(-1)
    return name.decode()


def bump_kv_lens(vnode_to_kv_lens, last_vnodes):
    """``vnode_to_kv_lens[last_vnodes] += 1`` on the device, current stream."""
    _table("vnode_to_kv_lens", vnode_to_kv_lens)
    _table("last_vnodes", last_vnodes)
    stream = torch.cuda.current_stream(vnode_to_kv_lens.device).cuda_stream
    _lib.check(_lib.load().ft_bump_kv_lens(vnode_to_kv_lens.data_ptr(), last_vnodes.data_ptr(),
                                           last_vnodes.numel(), stream))


def gather_kv_entries(src_table, seg_src, seg_len, seg_dst, seg_room, n_segments, aux_table):
    """Build the auxiliary row-id table on the device (``ft_gather_kv_entries``): segment ``i`` copies
    ``seg_len[i]`` ids from ``src_table[seg_src[i]:]`` to ``aux_table[seg_dst[i]:]`` and pads ``seg_room[i]``
    entries behind them with the segment's first id.  All tensors int32 on one CUDA device; current stream."""
    for name, t in (("src_table", src_table), ("seg_src", seg_src), ("seg_len", seg_len), ("seg_dst", seg_dst),
                    ("seg_room", seg_room), ("aux_table", aux_table)):
        _table(name, t)
    if min(seg_src.numel(), seg_len.numel(), seg_dst.numel(), seg_room.numel()) < n_segments:
        raise ValueError("segment tables are shorter than n_segments")
    stream = torch.cuda.current_stream(aux_table.device).cuda_stream
    _lib.check(_lib.load().ft_gather_kv_entries(src_table.data_ptr(), src_table.numel(), seg_src.data_ptr(),
                                                seg_len.data_ptr(), seg_dst.data_ptr(), seg_room.data_ptr(),
                                                int(n_segments), aux_table.data_ptr(), aux_table.numel(), stream))


def bump_tails(tail_state, n, row_ranges, vnode_to_kv_lens):
    """One step of a burst (``ft_bump_tails``): per request, either the grouped tail's partial row sees one
    token more (its range end in ``row_ranges`` moves up), or the tail's own vnode grows by one.
    ``tail_state`` is an int32 ``[n, 4]`` CUDA tensor ``{aux_pos | -1, src_pos, partial row | vnode, room}``."""
    _table("tail_state", tail_state)
    _table("vnode_to_kv_lens", vnode_to_kv_lens)
    if tail_state.numel() < 4 * n:
        raise ValueError("tail_state is shorter than 4 * n")
    if row_ranges is not None:
        _table("row_ranges", row_ranges)
    stream = torch.cuda.current_stream(tail_state.device).cuda_stream
    _lib.check(_lib.load().ft_bump_tails(
        tail_state.data_ptr(), int(n), row_ranges.data_ptr() if row_ranges is not None else None,
        row_ranges.numel() // 2 if row_ranges is not None else 0, vnode_to_kv_lens.data_ptr(), vnode_to_kv_lens.numel(),
        stream))


def refresh_tails(tail_state, n, src_table, aux_table):
    """``aux_table[aux_pos - 1] = src_table[src_pos - 1]`` for every grouped tail (``ft_refresh_tails``): the
    newest token's row id, which exists only once the step's batch has been prepared.  Current stream."""
    for name, t in (("tail_state", tail_state), ("src_table", src_table), ("aux_table", aux_table)):
        _table(name, t)
    if tail_state.numel() < 4 * n:
        raise ValueError("tail_state is shorter than 4 * n")
    stream = torch.cuda.current_stream(tail_state.device).cuda_stream
    _lib.check(_lib.load().ft_refresh_tails(tail_state.data_ptr(), int(n), src_table.data_ptr(), src_table.numel(),
                                            aux_table.data_ptr(), aux_table.numel(), stream))
