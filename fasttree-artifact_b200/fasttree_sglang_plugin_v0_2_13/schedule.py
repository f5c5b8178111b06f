"""Host planner of the plugin (reference:
fasttree_sglang_plugin_v0_2_13/schedule.py:12-283).

``prepare_for_fasttree_meta`` turns the running batch and SGLang's radix cache
into vnode tables addressed THROUGH ``req_to_token``: a tree vnode's KV run is
``stride * req_pool_idx[first request] + token offset`` into the flattened
table, which the kernels dereference to KV-pool slots.  Every request also gets
private "tail" vnodes over the positions the radix cache does not hold
(generated tokens and the token being decoded).  ``prepare_for_fasttree_step``
lengthens each request's last tail vnode by one between the steps of a burst.

Two planners, selected by ``FastTreeMetadata.planner``:

* ``"reference"`` reproduces the reference's tables bit for bit, including its
  quirks (the edge heuristic never fires because the child loop iterates over
  ``enumerate`` tuples, schedule.py:96-98; the 128-token KV-split fallback is a
  no-op, :130; a tile-size collapse copies the REQUEST tile into the KV tile
  sizes, :138-141; CTA counting uses the KV tile, not the split, :115; head
  counts are the unsharded ones).
* ``"b200"`` plans with the 148-SM splitter of ``ft_b200.planner`` (working edge
  decisions, chunk sizes from a byte budget, 128-row tiles for the tcgen05
  kernel) and starts each tail where the radix walk actually stopped, so prompt
  tokens that are not in the cache are still attended to.
"""
from collections import deque

import numpy as np
import torch

from ft_b200 import engine as _engine
from ft_b200 import planner as _planner


def _walk_requests(batch):
    """Per request, follow the radix tree along prompt + generated tokens
    (schedule.py:18-35).  Returns (node -> request ids, tokens covered per request)."""
    root = batch.tree_cache.root_node
    seen = {}           # node -> (request ids, tokens)
    covered = []
    for rid, req in enumerate(batch.reqs):
        prompt, output = req.origin_input_ids, req.output_ids
        n_prompt = len(prompt)
        n_tokens = n_prompt + len(output)
        node, pos = root, 0
        while pos < n_tokens:
            child = node.children.get(prompt[pos] if pos < n_prompt else output[pos - n_prompt])
            if not child:
                break
            entry = seen.get(child)
            if entry is None:
                entry = seen[child] = ([], len(child.key))
            entry[0].append(rid)
            node = child
            pos += entry[1]
        covered.append(pos)
    return {node: reqs for node, (reqs, _) in seen.items()}, covered


def _length(value):
    """Entries of a radix node's value: a 1-D tensor, or a list (a tensor's ``len`` costs a microsecond per node)."""
    return value.numel() if isinstance(value, torch.Tensor) else len(value)


def _bfs(batch, node_to_reqs):
    """Populated radix nodes in breadth-first order with their token offsets, parents and lengths (schedule.py:74-85)."""
    order, offsets, parents, lens = [], [], [], []
    todo = deque([(batch.tree_cache.root_node, 0, -1)])
    while todo:
        node, off, par = todo.popleft()
        me = len(order)
        order.append(node)
        offsets.append(off)
        parents.append(par)
        lens.append(_length(node.value))
        nxt = off + lens[me]
        for child in node.children.values():
            if child in node_to_reqs:
                todo.append((child, nxt, me))
    return order, offsets, parents, lens


def _upload(md, tabs, last_vnodes, tail_state=None, src_table=None):
    nv, rows, bsz = tabs["vnode_to_kv_offs"].size, tabs["vnode_to_q_entries"].size, tabs["req_to_vnode_offs"].size
    if nv > md.max_vnodes or rows > md.max_vnode_to_q_entries or bsz > md.max_batch_size:
        raise ValueError(f"plan ({nv} vnodes, {rows} partial rows, batch {bsz}) exceeds the capacity of "
                         f"FastTreeMetadata ({md.max_vnodes}, {md.max_vnode_to_q_entries}, {md.max_batch_size})")
    segs = tabs.get("aux_segments")
    n_seg = 0 if segs is None else int(segs.shape[0])
    if getattr(md, "group_tails", False):
        if n_seg > md.aux_segments.shape[1] or int(tabs.get("aux_entries", 0)) > md.kv_entries_aux.numel():
            raise ValueError(f"plan ({n_seg} grouped runs, {tabs.get('aux_entries', 0)} auxiliary row ids) exceeds the "
                             f"capacity of FastTreeMetadata ({md.aux_segments.shape[1]}, {md.kv_entries_aux.numel()})")

    def put(dst, arr):
        t = torch.from_numpy(np.ascontiguousarray(arr, dtype=np.int32))
        dst[:t.numel()].copy_(t, non_blocking=True)

    put(md.vnode_to_q_entries, tabs["vnode_to_q_entries"])
    put(md.vnode_to_q_offs, tabs["vnode_to_q_offs"])
    put(md.vnode_to_q_lens, tabs["vnode_to_q_lens"])
    put(md.vnode_to_kv_offs, tabs["vnode_to_kv_offs"])
    put(md.vnode_to_kv_lens, tabs["vnode_to_kv_lens"])
    put(md.req_to_vnode_entries, tabs["req_to_vnode_entries"])
    put(md.req_to_vnode_offs, tabs["req_to_vnode_offs"])
    put(md.req_to_vnode_lens, tabs["req_to_vnode_lens"])
    put(md.req_last_vnodes_dev, np.asarray(last_vnodes, dtype=np.int32))
    put(md.phase_info_dev, np.asarray(list(tabs["phase_node_nums"]) + list(tabs["phase_node_offsets"]), dtype=np.int32))
    state = np.full((bsz, 4), -1, dtype=np.int32)
    if tail_state is None:                      # every tail is a vnode of its own
        state[:, 2] = np.asarray(last_vnodes, dtype=np.int32)
    else:
        state[:] = tail_state
    md.tail_state[:bsz].copy_(torch.from_numpy(state), non_blocking=True)
    stale = getattr(md, "tail_rows", 0)
    if stale > bsz:                             # entries of a larger earlier batch must read "unused"
        md.tail_state[bsz:stale].fill_(-1)
    md.tail_rows = bsz
    md.num_grouped_tails = int((state[:, 0] >= 0).sum())
    md.steps_since_plan = 0
    if getattr(md, "group_tails", False):
        # the decode call always passes the range table: rows of plain vnodes see their whole chunk
        ranges = tabs.get("vnode_q_kv_ranges")
        if ranges is None:
            ranges = np.zeros((rows, 2), dtype=np.int32)
            ranges[:, 1] = np.iinfo(np.int32).max
        md.vnode_q_kv_ranges[:rows].copy_(torch.from_numpy(np.ascontiguousarray(ranges, dtype=np.int32)), non_blocking=True)
        if n_seg:
            md.aux_segments[:, :n_seg].copy_(torch.from_numpy(np.ascontiguousarray(segs.T, dtype=np.int32)), non_blocking=True)
            if md.kv_entries_aux.is_cuda:
                _engine.gather_kv_entries(src_table, md.aux_segments[0], md.aux_segments[1], md.aux_segments[2],
                                          md.aux_segments[3], n_seg, md.kv_entries_aux)
            else:       # plan tables kept on the host (planner tests, tools): the same table, built with torch
                flat = src_table.reshape(-1)
                for src, length, dst, room in segs.tolist():
                    md.kv_entries_aux[dst:dst + length] = flat[src:src + length]
                    md.kv_entries_aux[dst + length:dst + length + room] = flat[src]
        md.refresh_pending = md.num_grouped_tails > 0 or (md.graph_safe and md.refresh_layer is None)
    md.phase_node_nums = list(tabs["phase_node_nums"])
    sizes = tabs.get("task_sizes") or _planner.task_sizes(tabs["phase_node_nums"], tabs["vnode_to_kv_lens"],
                                                          tabs["vnode_to_q_lens"], md.kv_group_num)
    # The plan's rows, far fewer than the buffers': the merge kernel is chosen by their number (512 requests 13 270 ->
    # 13 150 us per burst).  A captured step has to fit every later plan and to give what an eager call gives: six rows per
    # request, which for few requests picks the form that is never far behind (us per step, the buffers' rows / six stated:
    # 12 requests of 3 rows at 32/8 heads 12.9 / 11.5, 24 of 6 at 28/4 14.7 / 11.4, 12 of 25 at 28/4 14.9 / 15.1).
    sizes = (*sizes, 6 * int(bsz) if md.graph_safe else int(rows))
    md.vnode_to_kv_lens.task_sizes = sizes
    md.phase_node_offsets = list(tabs["phase_node_offsets"])
    md.req_last_vnodes = [int(v) for v in last_vnodes]
    md.num_vnodes, md.num_partial_rows = int(nv), int(rows)


# --------------------------------------------------------------- reference-compatible
def _plan_reference(batch, md, node_to_reqs, order, offsets, lens, req_idx, stride):
    tsq, tsk = list(md.TSQs), list(md.TSKs)
    split = [md.kv_split_sizes[0], md.kv_split_sizes[0]]
    heads = md.num_kv_heads
    counts = [len(node_to_reqs[n]) if n in node_to_reqs else 0 for n in order]

    def cta_counts():                                   # schedule.py:87-118 with the heuristic inert
        par = [0, 0]
        for cnt, ln in zip(counts, lens):
            if cnt > 0:
                ph = 0 if cnt > tsq[1] else 1
                par[ph] += -(-cnt // tsq[ph]) * -(-ln // tsk[ph])
        return [c * heads for c in par]

    for rnd in range(3):                                # schedule.py:120-143
        par = cta_counts()
        if rnd == 0:
            if not any(0 < par[ph] < md.para_threshs1[ph] for ph in range(2)):
                break                                    # (the split-size assignment of the reference is a no-op)
        elif rnd == 1:
            if 0 < par[0] < md.para_threshs2[0]:
                tsq = [tsq[1], tsq[1]]
                tsk = [tsq[1], tsq[1]]
            elif 0 < par[1] < md.para_threshs2[1]:
                tsq = [tsq[0], tsq[0]]
                tsk = [tsq[0], tsq[0]]
            else:
                break
    md.phase_q_tile_sizes, md.phase_kv_tile_sizes = tsq, tsk

    vnodes = []
    for node, cnt, ln, off in zip(order, counts, lens, offsets):            # schedule.py:159-210
        if cnt == 0:
            continue
        kids = [c for c in node.children.values() if c in node_to_reqs]
        group = kids if kids else [node]
        reqs = [r for n in group for r in node_to_reqs[n]]
        first = node_to_reqs[group[0]][0]
        start = stride * req_idx[first] + off
        ph = 0 if cnt > tsq[1] else 1
        # the reference sizes the request tiles from `cnt` but lists `reqs`; they agree whenever
        # every request of a node continues into one of its children (true for its workloads)
        if len(reqs) != cnt:
            raise ValueError("a request ends exactly at an inner radix node; the reference planner's tables are "
                             "inconsistent for such batches (use planner='b200')")
        vnodes.append(_planner.VirtualNode([(start, start + ln)], np.asarray(reqs, dtype=np.int32),
                                           q_tile=tsq[ph], kv_split=split[ph]))
    tails = []
    for rid, req in enumerate(batch.reqs):                                  # schedule.py:212-232
        start = stride * req_idx[rid] + len(req.origin_input_ids)
        tails.append(_planner.VirtualNode([(start, start + len(req.output_ids) + 1)],
                                          np.asarray([rid], dtype=np.int32), q_tile=tsq[1], kv_split=split[1]))
    perm = []
    tabs = _planner.emit_tables(vnodes + tails, len(batch.reqs), small_tile=tsq[1], direct_offsets=True,
                                order_out=perm)
    # tail tasks are the last ones before and after the stable phase split: each request's last chunk
    n_tasks = tabs["vnode_to_kv_offs"].size
    last, acc = [], n_tasks - sum(-(-(len(r.output_ids) + 1) // split[1]) for r in batch.reqs)
    for req in batch.reqs:
        acc += -(-(len(req.output_ids) + 1) // split[1])
        last.append(acc - 1)
    tabs["req_to_vnode_entries"] = tabs["req_to_vnode_entries"][:-_planner.PAD_ENTRIES]   # the plugin uploads no padding
    return tabs, last


# ------------------------------------------------------------------------ B200 splitter
class _RadixView:
    """Radix node as the tree record the splitter expects."""
    __slots__ = ("parent", "id", "seqlen", "num_children", "requests")

    def __init__(self, parent, nid, seqlen, requests):
        self.parent, self.id, self.seqlen, self.num_children, self.requests = parent, nid, seqlen, 0, requests


def _plan_b200(batch, md, node_to_reqs, covered, order, offsets, parents, lens, req_idx, stride):
    model = _planner.b200_model_for(md, md.head_dim)
    all_reqs = list(range(len(batch.reqs)))
    tree = []
    for i, (node, par) in enumerate(zip(order, parents)):
        reqs = all_reqs if i == 0 else sorted(node_to_reqs[node])
        tree.append(_RadixView(par, i, lens[i], reqs))
        if par >= 0:
            tree[par].num_children += 1

    def ranges_of(assign, i):
        # a node and the ancestors it carries are one contiguous run in the row of any request below it
        start, up = offsets[i], i
        while assign[up] == 1:
            up = tree[up].parent
            start = offsets[up]
        first = tree[i].requests[0]
        base = stride * req_idx[first]
        return [(base + start, base + offsets[i] + tree[i].seqlen)]

    # Radix nodes that only one request passes through (the unique end of its prompt) are contiguous with that
    # request's tail in its row of req_to_token: they leave the tree and the tail starts where they began, which
    # makes one few-row task per request out of two or more.
    tail_start = list(covered)
    if getattr(md, "merge_private_nodes", True):
        for i in range(len(tree) - 1, 0, -1):      # children come after their parents in breadth-first order
            if len(tree[i].requests) == 1 and tree[i].num_children <= 1:
                rid = tree[i].requests[0]
                tail_start[rid] = min(tail_start[rid], offsets[i])
                tree[i].requests = []
                tree[tree[i].parent].num_children -= 1
    bsz = len(batch.reqs)
    rids = np.arange(bsz, dtype=np.int64)
    base = stride * np.asarray(req_idx, dtype=np.int64)
    tail_end = base + np.fromiter((len(r.origin_input_ids) + len(r.output_ids) + 1 for r in batch.reqs), dtype=np.int64, count=bsz)
    extra = np.stack([base + np.asarray(tail_start, dtype=np.int64), tail_end, rids], axis=1)
    native = getattr(md, "native_planner", True)
    if native:
        arrays = _planner._tree_arrays(tree)
        node_base = [stride * req_idx[nd.requests[0]] if nd.requests else 0 for nd in tree]

    def run(tail_room, model):
        if native:
            # the native splitter of the shared library; the Python branch below is its specification
            return _planner.b200_tables_native_direct(
                tree, node_base, offsets, extra, bsz, md.num_qo_heads, md.num_kv_heads, md.head_dim, model,
                tail_room=tail_room, arrays=arrays)
        vnodes, _assign, q_tile, small_tile, _target = _planner.b200_virtual_nodes(
            tree, md.num_qo_heads, md.num_kv_heads, md.head_dim, model, ranges_of,
            extra=[([(b, e)], [r]) for b, e, r in extra.tolist()], tail_room=tail_room)
        tabs = _planner.emit_tables(vnodes, len(batch.reqs), small_tile=small_tile, direct_offsets=True,
                                    order_key=_planner.b200_task_order)
        return tabs, q_tile, small_tile, model.tile_tokens

    # Every request has a few-row tail task of its own in a plan without groups: where those alone pass the bound below,
    # that plan would only be made to be replaced.
    bound = md.group_tails_min_load * model.num_sms * model.ctas_per_sm if getattr(md, "group_tails", False) else None
    tabs = None
    if bound is None or bsz * md.num_kv_heads < bound:
        tabs, q_tile, small_tile, tile_tokens = run(-1, model)
    if bound is not None:
        # Groups pay when the few-row tasks alone would queue up several deep behind the resident CTAs; then the
        # burst is planned with short runs packed into many-row vnodes.  A group needs more than 16 query
        # rows anyway (only the many-row kernels honour row ranges); past that, a handful of one-tile tails
        # already costs less as one task than as one task each.
        few_row_ctas = (bsz if tabs is None else tabs["phase_node_nums"][1]) * md.num_kv_heads
        if few_row_ctas >= bound:
            from dataclasses import replace
            tabs, q_tile, small_tile, tile_tokens = run(
                md.tail_room, replace(model, group_min_members=min(model.group_min_members, 4)))
    md.phase_q_tile_sizes = [q_tile, small_tile]
    md.phase_kv_tile_sizes = [tile_tokens, tile_tokens]
    # the task holding the END of each request's tail (the one that grows during the burst)
    last = np.full(bsz, -1, dtype=np.int64)
    kv_offs = tabs["vnode_to_kv_offs"].astype(np.int64)
    q_offs, q_lens, q_entries = tabs["vnode_to_q_offs"], tabs["vnode_to_q_lens"], tabs["vnode_to_q_entries"]
    single = np.flatnonzero((q_lens == 1) & (kv_offs < _planner.AUX_BIT))
    owner = q_entries[q_offs[single]]
    ends_tail = kv_offs[single] + tabs["vnode_to_kv_lens"][single] == tail_end[owner]
    last[owner[ends_tail]] = single[ends_tail]
    # tails that became members of a group: the run that ends where the request ends and has room behind it
    state = np.full((bsz, 4), -1, dtype=np.int32)
    segs = tabs.get("aux_segments")
    if segs is not None and len(segs):
        segs = segs.astype(np.int64)
        by_end = np.argsort(tail_end)
        at = np.minimum(np.searchsorted(tail_end[by_end], segs[:, 0] + segs[:, 1]), bsz - 1)
        rid = by_end[at]
        tails = (tail_end[rid] == segs[:, 0] + segs[:, 1]) & (segs[:, 3] > 0)
        rid, (src, length, dst, room) = rid[tails], segs[tails].T
        groups = np.flatnonzero(kv_offs >= _planner.AUX_BIT)
        groups = groups[np.argsort(kv_offs[groups], kind="stable")]
        member_of = np.searchsorted(kv_offs[groups] - _planner.AUX_BIT, dst, side="right") - 1
        # the groups' partial rows as (group, request) keys: a grouped tail has exactly one
        g_len = q_lens[groups].astype(np.int64)
        g_start = np.cumsum(g_len) - g_len
        rows = np.arange(int(g_len.sum())) + np.repeat(q_offs[groups] - g_start, g_len)
        keys = np.repeat(np.arange(groups.size), g_len) * bsz + q_entries[rows]
        by_key = np.argsort(keys, kind="stable")
        want = member_of * bsz + rid
        lo, hi = (np.searchsorted(keys[by_key], want, side=side) for side in ("left", "right"))
        if np.any(hi - lo != 1):
            raise RuntimeError("internal error: a grouped tail has no partial row of its own")
        state[rid] = np.stack([dst + length, src + length, rows[by_key[lo]], room], axis=1)
        last[rid] = groups[member_of]
    if bsz and last.min() < 0:
        raise RuntimeError("internal error: a request has no tail task")
    own = state[:, 0] < 0
    state[own, 2] = last[own]
    tabs["req_to_vnode_entries"] = tabs["req_to_vnode_entries"][:-_planner.PAD_ENTRIES]
    tabs["tail_state"] = state
    return tabs, last


def prepare_for_fasttree_meta(batch, fasttree_metadata):
    """Plan one decode burst and upload the tables into ``fasttree_metadata``
    (reference: schedule.py:12-275).  Binds the metadata to the batch."""
    md = fasttree_metadata
    node_to_reqs, covered = _walk_requests(batch)
    order, offsets, parents, lens = _bfs(batch, node_to_reqs)
    # one row of the table per request; a tensor padded beyond the batch is fine, one that is too short is not
    bsz = len(batch.reqs)
    req_idx = batch.req_pool_indices.tolist()[:bsz]
    if bsz and not isinstance(req_idx[0], int):         # one index per row, or floats
        req_idx = [int(i) for i in batch.req_pool_indices[:bsz].reshape(-1).tolist()]
    if len(req_idx) != bsz:
        raise IndexError(f"req_pool_indices names {len(req_idx)} of {bsz} requests")
    stride = batch.req_to_token_pool.req_to_token.stride(0)
    if md.planner == "reference":
        tabs, last = _plan_reference(batch, md, node_to_reqs, order, offsets, lens, req_idx, stride)
    else:
        tabs, last = _plan_b200(batch, md, node_to_reqs, covered, order, offsets, parents, lens, req_idx, stride)
    _upload(md, tabs, last, tail_state=tabs.get("tail_state"),
            src_table=batch.req_to_token_pool.req_to_token if getattr(md, "group_tails", False) else None)
    batch.fasttree_metadata = md


def prepare_for_fasttree_step(batch, fasttree_metadata):
    """Between two steps of a burst: the token just decoded joins each request's
    last private chunk (reference: schedule.py:278-283).  One tiny kernel, no
    host-to-device copy."""
    md = fasttree_metadata
    md.steps_since_plan += 1
    if md.num_grouped_tails and md.steps_since_plan > md.tail_room:
        raise RuntimeError(f"a burst of more than {md.tail_room} steps after one plan: raise FastTreeMetadata.tail_room")
    if md.tail_state.is_cuda:
        _engine.bump_tails(md.tail_state, len(batch.reqs), md.vnode_q_kv_ranges, md.vnode_to_kv_lens)
    else:               # plan tables kept on the host (planner tests, tools)
        for rid in range(len(batch.reqs)):
            aux_pos, _src, index, room = md.tail_state[rid].tolist()
            if aux_pos < 0:
                md.vnode_to_kv_lens[index] += 1
            else:
                md.vnode_q_kv_ranges[index, 1] += 1
                md.tail_state[rid] += torch.tensor([1, 1, 0, -1], dtype=torch.int32)
    md.refresh_pending = md.num_grouped_tails > 0
