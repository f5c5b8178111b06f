"""The work that performance is measured on: decode steps of tree attention through the public entry points.

Three ways in, as a user's program takes them:

* ``tree``   plan once with ``fasttree_preparation``, then one ``fasttree_decode`` per decode step and layer: the
             micro-benchmark's loop, launched eagerly, everything resident on the GPU;
* ``host``   the same step with the query and the output in pinned host memory (``fasttree_decode_host_io``), as a
             decode loop whose sampler lives on the host calls it;
* ``serve``  a whole burst of the SGLang v0.2.13 plugin: re-plan from the radix cache, then a number of decode steps
             through every layer's patched ``RadixAttention.decode_forward``, either launched eagerly or, with the
             plan-independent launch (``graph_safe``), as one CUDA-graph replay per step.

``listed()`` are fixed cases from the repository's own configurations, tests and benchmark grid; ``draw(rng)`` gives
more of the same ranges.  Inputs are N(0, 1) tensors (Q scaled by 0.5 in bf16, as in the benchmark), made from the
seed on the GPU; one decode token per request.
"""
import os
import sys
import types

import torch

_PKG = os.path.abspath("fasttree-artifact_b200")      # the working folder is the repository's root
for _p in (_PKG, os.path.join(_PKG, "kernel_bench")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

import fasttree              # noqa: E402
import kv_tree_simple        # noqa: E402
import tree_generation       # noqa: E402

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}


def _tree(name, sizes, lens, hq, hkv, d, dtype, way="tree"):
    return {"name": name, "way": way, "sizes": sizes, "lens": lens, "hq": hq, "hkv": hkv, "d": d, "dtype": dtype}


def _serve(name, sizes, lens, generated, hq, hkv, dtype, layers, steps, layout, graph):
    return {"name": name, "way": "serve", "sizes": sizes, "lens": lens, "generated": generated, "hq": hq, "hkv": hkv,
            "d": 128, "dtype": dtype, "layers": layers, "steps": steps, "layout": layout, "graph": graph}


def listed():
    return [
        # the smallest configuration, in fp32: four requests, a few hundred tokens; latency of one call
        _tree("fp32_small", "1,4", "512,64", 8, 2, 128, "fp32"),
        # one KV head left on the GPU (a head-sharded rank, or the benchmark grid's 16/1 heads), ten requests
        _tree("one_kv_head", "1,10", "4000,400", 16, 1, 128, "fp16"),
        # the headline: 64 requests under one system prompt
        _tree("prefix_64", "1,64", "4096,256", 32, 8, 128, "fp16"),
        # the headline's step with the sampler on the host: query and output cross PCIe in every step
        _tree("prefix_64_host", "1,64", "4096,256", 32, 8, 128, "fp16", way="host"),
        # few-shot prompts over a shared preamble, many short questions under each
        _tree("three_levels_256", "1,16,256", "2048,512,64", 32, 8, 128, "bf16"),
        # extreme sharing: a thousand samples of one long context, tensor-bound
        _tree("prefix_1024", "1,1024", "16384,32", 64, 8, 128, "bf16"),
        # an irregular tree of uneven nodes (ragged lengths everywhere), the largest in bytes
        {"name": "random_6_levels", "way": "tree", "levels": 6, "tree_seed": 0, "hq": 32, "hkv": 8, "d": 128, "dtype": "fp16"},
        # a search tree: nine levels, mostly of 16-token nodes, no head grouping
        _tree("deep_short_nodes", "1,2,4,8,16,32,64,128,1024", "256,128,64,16,16,16,16,16,16", 32, 32, 128, "fp16"),
        # small heads (head_dim 64), four levels of the benchmark grid
        _tree("head_dim_64", "1,4,16,512", "1024,256,128,32", 32, 8, 64, "bf16"),
        # large heads (head_dim 256)
        _tree("head_dim_256", "1,64", "4096,256", 16, 8, 256, "bf16"),
        # serving: four system prompts with 128 questions each, pool slots scattered, eager launches, the burst
        # length SGLang v0.2.13 runs
        _serve("serve_system", "1,4,512", "24,420,36", "2,0,7,1", 32, 8, "fp16", 16, 10, "scattered", False),
        # serving: sixteen documents with eight questions each, the pool as prefill leaves it, one graph per step
        _serve("serve_documents_graph", "1,16,128", "12,1500,25", "1,4,0", 32, 8, "fp16", 16, 10, "prefill", True),
    ]


# ---------------------------------------------------------------------------------------------------- drawn cases
def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


_HEADS = ((32, 8), (32, 8), (32, 8), (64, 8), (32, 32), (16, 1), (8, 2), (4, 1), (24, 8), (28, 4), (16, 16))


def _draw_once(rng):
    way = rng.choices(("tree", "host", "serve"), (0.74, 0.08, 0.18))[0]
    hq, hkv = rng.choice(_HEADS)
    dtype = rng.choice(("fp16", "bf16"))
    if way == "serve":
        branches = _log_uniform(rng, 1, 32)
        per = _log_uniform(rng, 2, max(2, 512 // branches))
        graph = rng.random() < 0.4
        return {"way": way, "sizes": "1,%d,%d" % (branches, branches * per),
                "lens": "%d,%d,%d" % (_log_uniform(rng, 4, 256), _log_uniform(rng, 30, 1500), _log_uniform(rng, 8, 128)),
                "generated": ",".join(str(rng.randrange(12)) for _ in range(rng.randrange(2, 6))),
                "hq": hq, "hkv": hkv, "d": 128, "dtype": dtype, "layers": rng.randrange(4, 17),
                "steps": rng.randrange(4, 11), "layout": rng.choice(("scattered", "prefill")), "graph": graph}
    d = rng.choices((128, 64, 256), (0.62, 0.22, 0.16))[0]
    if way == "tree" and d != 256 and rng.random() < 0.1:
        dtype = "fp32"
    case = {"way": way}
    if rng.random() < 0.25:
        case.update(levels=rng.randrange(3, 7), tree_seed=rng.randrange(1 << 16))
    else:
        depth = rng.randrange(2, 6)
        leaves = _log_uniform(rng, 2, 1024)
        sizes = [1] + sorted(_log_uniform(rng, 1, leaves) for _ in range(depth - 2)) + [leaves]
        lens = [_log_uniform(rng, 16, 16384)] + [_log_uniform(rng, 8, 2048) for _ in range(depth - 2)]
        lens.append(_log_uniform(rng, 8, 1024))
        case.update(sizes=",".join(map(str, sizes)), lens=",".join(map(str, lens)))
    case.update(hq=hq, hkv=hkv, d=d, dtype=dtype)
    return case


def draw(rng):
    # no more work than the largest listed case of the same kind
    while True:
        case = _draw_once(rng)
        w = work(case)
        if case["way"] == "serve":
            limit = 1.4e10, 1e12
        elif case["dtype"] == "fp32":
            limit = 6e7, 1.2e9
        elif case["d"] == 256:
            limit = 1.8e8, 4.6e9
        elif case["way"] == "host":
            limit = 3e8, 5e10
        else:
            limit = 3.2e9, 5.6e11
        if w["bytes"] <= limit[0] and w["flops"] <= limit[1]:
            return case


# ------------------------------------------------------------------------------------------------------ the trees
def _ints(text):
    return [int(x) for x in text.split(",")]


def _nodes(case):
    """The case's tree with its requests assigned (leaves in id order), the batch size and the row offsets."""
    if "levels" in case:
        rows = tree_generation.generate_random_tree(case["levels"], case["tree_seed"])
    else:
        rows = tree_generation.generate_tree(_ints(case["sizes"]), _ints(case["lens"]))
    nodes = kv_tree_simple.tree_from_rows(rows)
    batch, ptrs = kv_tree_simple.assign_requests(nodes)
    return nodes, batch, ptrs


def _generated(case, batch):
    cycle = _ints(case["generated"])
    return [cycle[r % len(cycle)] for r in range(batch)]


def work(case):
    """Each K/V row of the tree and each query read once, each output written once; two products per (row, token)."""
    nodes, batch, ptrs = _nodes(case)
    hq, hkv, d = case["hq"], case["hkv"], case["d"]
    esize = 4 if case["dtype"] == "fp32" else 2
    tokens, pairs, calls = ptrs[-1], sum(n.seqlen * len(n.requests) for n in nodes), 1
    if case["way"] == "serve":      # plus every request's own tokens; as many calls as layers and steps
        own = sum(_generated(case, batch)) + batch * (case["steps"] + 1) / 2
        tokens, pairs, calls = tokens + own, pairs + own, case["layers"] * case["steps"]
    return {"bytes": calls * (2 * tokens * hkv * d * esize + 2 * batch * hq * d * esize), "flops": calls * 4 * d * hq * pairs}


def tolerance(case):
    # about four times what the present code is off by against the same attention in fp64 on these inputs:
    # fp16 rel 2.5e-4 .. 2.9e-4, max 1.5e-3; bf16 rel 2.4e-3, max 1.1e-2 (probabilities and outputs are rounded to the
    # storage type); fp32 rel 4e-7, max 4e-6
    return {"fp16": {"rel": 1.2e-3, "max": 6e-3}, "bf16": {"rel": 1e-2, "max": 4e-2},
            "fp32": {"rel": 2e-6, "max": 1.6e-5}}[case["dtype"]]


# ------------------------------------------------------------------------------------------------------ one pass
def prepare(case, seed):
    return _prepare_serve(case, seed) if case["way"] == "serve" else _prepare_tree(case, seed)


def run(state):
    return state["pass"](state)


def _randn(gen, *shape, dtype, scale=1.0):
    out = torch.empty(shape, dtype=dtype, device="cuda")
    flat = out.view(-1)
    step = 1 << 26      # in blocks: the fp32 draws of a large pool would not be small beside it
    for at in range(0, flat.numel(), step):
        part = flat[at:at + step]
        part.copy_(torch.randn(part.numel(), generator=gen, device="cuda").mul_(scale))
    return out


def _prepare_tree(case, seed):
    dtype, hq, hkv, d = DTYPES[case["dtype"]], case["hq"], case["hkv"], case["d"]
    nodes, batch, ptrs = _nodes(case)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    k = _randn(gen, ptrs[-1], hkv, d, dtype=dtype)
    v = _randn(gen, ptrs[-1], hkv, d, dtype=dtype)
    q = _randn(gen, batch, hq, d, dtype=dtype, scale=0.5 if case["dtype"] == "bf16" else 1.0)
    o = torch.empty_like(q)
    params = fasttree.FastTreeParams()
    group = hq // hkv
    params.set_kv_group_num(group)
    params.set_q_tile_sizes([max(1, 64 // group), max(1, 16 // group)])
    params.set_kv_tile_sizes([32, 32])
    params.set_kv_dtype(dtype)
    aux, _ = fasttree.fasttree_preparation(nodes, ptrs, batch, hq, hkv, d, [1024, 128], [132, 528], [132, 132], params)
    state = {"k": k, "v": v, "aux": aux, "tsq": params.TSQs, "tsk": params.TSKs, "scale": d ** -0.5}
    if case["way"] == "host":
        state["q"] = q.cpu().pin_memory()
        state["o"] = o.cpu().pin_memory()
        state["pass"] = _host_step
    else:
        state["q"], state["o"] = q, o
        state["pass"] = _tree_step
    return state


def _tree_step(s):
    fasttree.fasttree_decode(s["q"], s["k"], s["v"], s["o"], *s["aux"], s["tsq"], s["tsk"], s["scale"])
    return s["o"]


def _host_step(s):
    fasttree.fasttree_decode_host_io(s["q"], s["k"], s["v"], s["o"], *s["aux"], s["tsq"], s["tsk"], s["scale"])
    return s["o"]


# ------------------------------------------------------------------------------------------- the serving host
# SGLang v0.2.13 is not installed here: these classes hold what the plugin reads of it and behave as it does on this
# path - radix nodes of token ids and pool slots, a request-to-slot table whose newest entries are written when a
# step's batch is prepared, one K/V pool per layer.
class _RadixNode:
    def __init__(self, parent, key, value):
        self.parent, self.key, self.value, self.children = parent, key, value, {}


class _RadixAttention:
    def __init__(self, num_heads, head_dim, scaling, num_kv_heads, layer_id, logit_cap=-1):
        self.tp_q_head_num, self.tp_k_head_num = num_heads, num_kv_heads
        self.qk_head_dim = self.v_head_dim = head_dim
        self.scaling, self.layer_id, self.logit_cap = scaling, layer_id, logit_cap
        self.decode_forward = None

    def store_kv_cache(self, k, v, meta):
        pool, loc = meta.token_to_kv_pool, meta.out_cache_loc
        pool.get_key_buffer(self.layer_id)[loc] = k.view(-1, self.tp_k_head_num, self.qk_head_dim)
        pool.get_value_buffer(self.layer_id)[loc] = v.view(-1, self.tp_k_head_num, self.v_head_dim)


class _InputMetadata:
    @classmethod
    def from_schedule_batch(cls, model_runner, batch, forward_mode):
        self = cls()
        self.token_to_kv_pool, self.req_to_token_pool = batch.token_to_kv_pool, batch.req_to_token_pool
        self.out_cache_loc = batch.out_cache_loc
        return self


class _Batch:
    """A running batch: requests, radix cache, pools."""

    def is_empty(self):
        return not self.reqs

    def has_stream(self):
        return False


class _KVPool:
    def __init__(self, k, v):
        self.k, self.v = k, v

    def get_key_buffer(self, layer):
        return self.k[layer]

    def get_value_buffer(self, layer):
        return self.v[layer]


class _TpServer:
    """What the patched ``__init__`` and ``forward_step`` use of SGLang's worker."""

    def __init__(self, gpu_id, tp_rank, server_args, nccl_port, model_overide_args):
        self.gpu_id, self.tp_rank, self.model_config = gpu_id, tp_rank, model_overide_args
        self.running_batch, self.out_pyobjs = None, []
        self.num_generated_tokens = self.decode_forward_ct = 0

    def get_new_prefill_batch(self):
        return None

    def print_decode_stats(self):
        pass

    def forward_decode_batch(self, batch):
        self.decode_forward_ct += 1
        self.decode(batch)


_config = types.SimpleNamespace(num_continue_decode_steps=10, init_new_token_ratio=0.7)


def _install_host():
    if "sglang.srt.managers.tp_worker" in sys.modules:
        return
    for name, attrs in (("sglang", {}), ("sglang.srt", {}), ("sglang.srt.managers", {}), ("sglang.srt.layers", {}),
                        ("sglang.srt.model_executor", {}),
                        ("sglang.srt.managers.tp_worker", {"ModelTpServer": _TpServer, "global_config": _config}),
                        ("sglang.srt.layers.radix_attention", {"RadixAttention": _RadixAttention}),
                        ("sglang.srt.model_executor.forward_batch_info", {"InputMetadata": _InputMetadata})):
        mod = types.ModuleType(name)
        mod.__dict__.update(attrs)
        sys.modules[name] = mod
    from fasttree_sglang_plugin_v0_2_13 import load_fasttree_plugin
    load_fasttree_plugin()


def _prepare_serve(case, seed):
    _install_host()
    dtype, hq, hkv, d = DTYPES[case["dtype"]], case["hq"], case["hkv"], case["d"]
    layers, steps = case["layers"], case["steps"]
    nodes, bsz, ptrs = _nodes(case)
    generated = _generated(case, bsz)
    host_rng = torch.Generator().manual_seed(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)

    # pool slots: radix nodes in consecutive slots and decode tokens interleaved across the requests (prefill), or a
    # random permutation (a pool fragmented by long use)
    longest = max(generated) + steps
    pool = ptrs[-1] + bsz * longest + 8
    perm = torch.arange(pool, dtype=torch.int32)
    if case["layout"] == "scattered":
        perm = torch.randperm(pool, generator=host_rng).to(torch.int32)
    own = perm[ptrs[-1]:ptrs[-1] + bsz * longest].view(longest, bsz)         # step-major

    radix = []
    for nd in nodes:
        above = radix[nd.parent] if nd.parent >= 0 else None
        if above is None and nd.seqlen > 0:     # SGLang's root is empty; the tree's root is its only child
            above = _RadixNode(None, [], perm[:0])
            root = above
        node = _RadixNode(above, list(range(1000 + ptrs[nd.id], 1000 + ptrs[nd.id + 1])), perm[ptrs[nd.id]:ptrs[nd.id + 1]])
        above.children[node.key[0]] = node
        radix.append(node)
    batch = _Batch()
    batch.tree_cache = types.SimpleNamespace(root_node=root)
    batch.reqs, rows = [], []
    next_token = 1000 + ptrs[-1]
    for nd in nodes:
        if nd.num_children:
            continue
        chain, cur = [], nd.id
        while cur != -1:
            chain.append(cur)
            cur = nodes[cur].parent
        chain.reverse()
        r = len(batch.reqs)
        prompt = [t for n in chain for t in radix[n].key]
        output = list(range(next_token, next_token + generated[r]))
        next_token += generated[r]
        batch.reqs.append(types.SimpleNamespace(origin_input_ids=prompt, output_ids=output))
        rows.append(torch.cat([radix[n].value for n in chain] + [own[:generated[r], r]]))
    table = torch.zeros(bsz + 3, max(len(row) for row in rows) + steps + 8, dtype=torch.int32)
    pool_idx = torch.randperm(bsz + 3, generator=host_rng)[:bsz]
    for r, row in enumerate(rows):
        table[pool_idx[r], :len(row)] = row
    batch.req_to_token_pool = types.SimpleNamespace(req_to_token=table.cuda())
    batch.req_pool_indices = pool_idx.to(torch.int32).cuda()
    ends = torch.tensor([len(row) for row in rows])
    # per step: where each request's new token goes in the table and in the pool
    at = [(pool_idx.cuda(), (ends + i).cuda()) for i in range(steps)]
    new_slots = [torch.stack([own[generated[r] + i, r] for r in range(bsz)]).cuda() for i in range(steps)]
    batch.out_cache_loc = new_slots[0].long()       # static: a captured step reads it, the loop rewrites it
    batch.token_to_kv_pool = _KVPool(*([_randn(gen, pool, hkv, d, dtype=dtype) for _ in range(layers)] for _ in range(2)))
    q = _randn(gen, steps, layers, bsz, hq * d, dtype=dtype, scale=0.5)
    k_new = _randn(gen, layers, bsz, hkv * d, dtype=dtype)
    v_new = _randn(gen, layers, bsz, hkv * d, dtype=dtype)
    os.environ["FASTTREE_GRAPH_SAFE"] = "1" if case["graph"] else "0"
    worker = sys.modules["sglang.srt.managers.tp_worker"].ModelTpServer(
        torch.cuda.current_device(), 1, types.SimpleNamespace(tp_size=1, disable_cuda_graph=False), 0,
        types.SimpleNamespace(num_attention_heads=hq, num_key_value_heads=hkv, head_dim=d))
    os.environ.pop("FASTTREE_GRAPH_SAFE")
    info = sys.modules["sglang.srt.model_executor.forward_batch_info"].InputMetadata
    attn_class = sys.modules["sglang.srt.layers.radix_attention"].RadixAttention
    attn = [attn_class(hq, d, d ** -0.5, hkv, i) for i in range(layers)]
    worker.running_batch = batch
    state = {"pass": _burst, "worker": worker, "batch": batch, "lengths": generated, "steps": steps}

    def layers_of(step_q):
        meta = info.from_schedule_batch(None, batch, "decode")
        return [attn[i].decode_forward(step_q[i], k_new[i], v_new[i], meta) for i in range(layers)]

    if case["graph"]:
        from fasttree_sglang_plugin_v0_2_13 import schedule
        with torch.inference_mode():
            step_q = q[0].clone()
            batch.req_to_token_pool.req_to_token[at[0]] = new_slots[0]
            schedule.prepare_for_fasttree_meta(batch, worker.fasttree_metadata)
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                layers_of(step_q)
                side.synchronize()
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=side):
                    graph_out = torch.stack(layers_of(step_q))
            torch.cuda.current_stream().wait_stream(side)
        state["graph"] = graph

    def decode(running):
        i = state["step"]
        state["step"] = i + 1
        # the step's batch: every request's new token gets its slot
        running.req_to_token_pool.req_to_token[at[i]] = new_slots[i]
        running.out_cache_loc.copy_(new_slots[i])
        if case["graph"]:
            step_q.copy_(q[i])
            graph.replay()
            state["out"].append(graph_out.clone())
        else:
            state["out"].append(torch.stack(layers_of(q[i])))
        for req in running.reqs:        # the sampled token
            req.output_ids.append(7)

    worker.decode = decode
    return state


def _burst(s):
    """One ``forward_step`` of the worker: plan, then the burst's decode steps.  Returns every step's attention
    outputs ``[layers, requests, heads * head_dim]``."""
    _config.num_continue_decode_steps = s["steps"]
    s["step"], s["out"] = 0, []
    s["worker"].forward_step()
    for req, n in zip(s["batch"].reqs, s["lengths"]):      # the burst is taken back: the next pass decodes it again
        del req.output_ids[n:]
    return s["out"]
