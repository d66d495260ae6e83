"""Performance cases: the work users have this framework do, through its public entry points.

Eight kinds of work, each over a range of sizes:

``gcn_step``     one training step of a two-layer GCN on a whole graph (forward, loss, gradients of the weights)
``gcn_infer``    the forward pass of a two-layer GCN, no gradients
``minibatch``    neighbour sampling of one batch and a training step of a two-layer GCN on it
``spmm``         the weighted aggregation alone, forward or forward and backward
``appnp``        K-hop personalised propagation, forward and backward
``gat``          one attention layer, inference or training
``edge_ops``     the per-edge operators one by one, each with its backward
``convert``      an unsorted edge list to normalised CSC and CSR

``listed()`` names twelve of them, ``draw()`` gives more of the same ranges.  Graphs are R-MAT
(0.57, 0.19, 0.19, 0.05) folded onto the node count, or the log-normal in-degree graph of the attention
workload; nothing is downloaded.
"""
import math

import torch

import jittorgeometric_b200 as jg
from jittorgeometric_b200 import nn, ops, sampling, synth

# share of the mirrored R-MAT edges that are distinct pairs at the densities used here
_DISTINCT = 0.92


def listed():
    return [
        # the citation-graph training step: a few MB of data, all launches and latency
        {"name": "citation_step", "kind": "gcn_step", "graph": "citation", "nodes": 2708, "edges": 5278,
         "fin": 1433, "hidden": 256, "classes": 7},
        # full-graph training on a medium graph with an odd class count
        {"name": "medium_step", "kind": "gcn_step", "graph": "rmat", "nodes": 169984, "edges": 1200000,
         "fin": 100, "hidden": 256, "classes": 47},
        # sampled training: 1024 seeds, fanout 25 and 10, features gathered, one step
        {"name": "minibatch_step", "kind": "minibatch", "nodes": 1 << 19, "edges": 16 << 19, "seeds": 1024,
         "fan0": 25, "fan1": 10, "fin": 128, "hidden": 128, "classes": 64},
        # the narrow end of the aggregation sweep
        {"name": "spmm_narrow", "kind": "spmm", "nodes": 1 << 20, "edges": 32 << 20, "width": 32, "backward": False},
        # an ordinary width on a ragged graph, both directions
        {"name": "spmm_ordinary", "kind": "spmm", "nodes": 700001, "edges": 9000000, "width": 72, "backward": True},
        # the wide end of the aggregation sweep, the largest graph of the sweep
        {"name": "spmm_wide", "kind": "spmm", "nodes": 1 << 21, "edges": 32 << 21, "width": 256, "backward": False},
        # propagation with a teleport term, as a predict-then-propagate model trains it
        {"name": "appnp_train", "kind": "appnp", "nodes": 250007, "edges": 2500000, "width": 40, "hops": 10},
        # inference over a graph of millions of nodes, the widths of the partitioned workload
        {"name": "gcn_infer", "kind": "gcn_infer", "nodes": 1 << 22, "edges": 16 << 22, "fin": 128, "hidden": 128,
         "classes": 64},
        # the attention workload, training: 8 heads of 8 on a dense social-network-shaped graph, input width 602
        {"name": "gat_train", "kind": "gat", "nodes": 232965, "edges": 114600000, "fin": 602, "heads": 8, "dim": 8,
         "backward": True},
        # the reference's single-head attention layer, inference on a sparse graph
        {"name": "gat_infer", "kind": "gat", "nodes": 120000, "edges": 3000000, "fin": 128, "heads": 1, "dim": 64,
         "backward": False},
        # the operators an op-by-op attention model is built of, forward and backward
        {"name": "edge_ops", "kind": "edge_ops", "nodes": 29120, "edges": 7000000, "channels": 64, "heads": 8},
        # the conversion workload: shuffled R-MAT edge list with duplicates and a few loops, unit weights
        {"name": "convert_large", "kind": "convert", "nodes": 1 << 24, "edges": 16 << 24, "weighted": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gcn_step", "gcn_infer", "minibatch", "spmm", "appnp", "gat", "edge_ops", "convert"])
    if kind == "gcn_step":
        n = _log(rng, 2000, 400000)
        return {"kind": kind, "graph": "rmat", "nodes": n, "edges": int(n * rng.uniform(2, 16)), "fin": _log(rng, 16, 1433),
                "hidden": _log(rng, 16, 256), "classes": rng.randint(2, 64)}
    if kind == "gcn_infer":
        n = _log(rng, 1 << 16, 1 << 22)
        return {"kind": kind, "nodes": n, "edges": int(n * rng.uniform(4, 16)), "fin": rng.choice([64, 100, 128]),
                "hidden": rng.choice([32, 64, 128]), "classes": rng.randint(7, 64)}
    if kind == "minibatch":
        n = _log(rng, 1 << 16, 1 << 20)
        return {"kind": kind, "nodes": n, "edges": int(n * rng.uniform(8, 16)), "seeds": _log(rng, 128, 4096),
                "fan0": rng.randint(5, 25), "fan1": rng.randint(5, 15), "fin": _log(rng, 32, 256), "hidden": rng.choice([64, 128, 256]),
                "classes": rng.randint(7, 64)}
    if kind == "spmm":
        n = _log(rng, 1 << 14, 1 << 21)
        return {"kind": kind, "nodes": n, "edges": int(n * rng.uniform(4, 32)), "width": _log(rng, 7, 256),
                "backward": n < (1 << 20) and rng.random() < 0.5}
    if kind == "appnp":
        n = _log(rng, 1 << 14, 1 << 20)
        return {"kind": kind, "nodes": n, "edges": int(n * rng.uniform(4, 12)), "width": _log(rng, 7, 64), "hops": rng.choice([4, 10])}
    if kind == "gat":
        n = _log(rng, 10000, 232965)
        heads, dim = rng.choice([(1, 16), (1, 64), (2, 16), (4, 8), (4, 16), (8, 8), (8, 4)])
        return {"kind": kind, "nodes": n, "edges": int(n * math.exp(rng.uniform(math.log(10), math.log(492)))), "fin": _log(rng, 32, 602),
                "heads": heads, "dim": dim, "backward": rng.random() < 0.5}
    if kind == "edge_ops":
        n = _log(rng, 4000, 29120)
        return {"kind": kind, "nodes": n, "edges": int(n * math.exp(rng.uniform(math.log(10), math.log(240)))),
                "channels": rng.choice([16, 30, 64]), "heads": rng.choice([1, 4, 8])}
    n = _log(rng, 1 << 15, 1 << 23)
    return {"kind": kind, "nodes": n, "edges": int(n * rng.uniform(4, 16)), "weighted": rng.random() < 0.5}


# ------------------------------------------------------------------------------ inputs
def _rand_like(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape, device="cuda", generator=g)


def _rmat_edge_index(n, m, seed):
    """Symmetrised, deduplicated, relabelled R-MAT edges folded onto ``n`` nodes."""
    scale = max(1, (n - 1).bit_length())
    src, dst = synth.rmat_edges(scale, m, seed, device="cuda")
    return synth.symmetrise_dedupe(src % n, dst % n, n, relabel_seed=seed + 1)


def _attention_graph(case, seed):
    """The log-normal in-degree graph with exactly ``edges`` entries (cut, or the last column extended)."""
    E = case["edges"]
    rows, off = synth.lognormal_degree_csc(case["nodes"], int(1.03 * E), seed, device="cuda")
    if rows.numel() < E:
        rows = torch.cat([rows, rows[:E - rows.numel()]])
        off[-1] = E
    return jg.CSC(rows[:E].contiguous(), off.clamp(max=E), None)


def _normalised(case, seed):
    n = case["nodes"]
    if case.get("graph") == "citation":
        ei = synth.preferential_attachment(n, case["edges"], seed).cuda()
    else:
        ei = _rmat_edge_index(n, case["edges"], seed)
    return jg.gcn_norm_csc_csr(ei, None, n)


def _features(case, seed):
    n, f = case["nodes"], case["fin"]
    if case.get("graph") == "citation":
        return synth.sparse_binary_features(n, f, 18, seed, device="cuda")
    return _rand_like((n, f), seed)


def _labels(n, classes, seed):
    return torch.randint(classes, (n,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))


def _two_layers(case, seed):
    torch.manual_seed(seed)
    return (nn.GCNConv(case["fin"], case["hidden"], relu=True).cuda(), nn.GCNConv(case["hidden"], case["classes"]).cuda())


def prepare(case, seed):
    kind, n = case["kind"], case["nodes"]
    s = {"case": case}
    if kind in ("gcn_step", "gcn_infer"):
        s["csc"], s["csr"] = _normalised(case, seed)
        s["x"] = _features(case, seed + 100)
        s["labels"] = _labels(n, case["classes"], seed + 200)
        s["conv1"], s["conv2"] = _two_layers(case, seed)
    elif kind == "minibatch":
        s["csc"] = jg.cootocsc(_rmat_edge_index(n, case["edges"], seed), None, n)
        s["x"] = _rand_like((n, case["fin"]), seed + 100)
        s["labels"] = _labels(n, case["classes"], seed + 200)
        g = torch.Generator(device="cuda").manual_seed(seed + 300)
        s["seeds"] = torch.randperm(n, device="cuda", generator=g)[:case["seeds"]].to(torch.int32)
        s["conv1"], s["conv2"] = _two_layers(case, seed)
        s["seed"] = seed
    elif kind == "spmm":
        s["csc"], s["csr"] = _normalised(case, seed)
        s["x"] = _rand_like((n, case["width"]), seed + 100).requires_grad_(case["backward"])
        s["gy"] = _rand_like((n, case["width"]), seed + 200) if case["backward"] else None
    elif kind == "appnp":
        s["csc"], s["csr"] = _normalised(case, seed)
        s["x"] = _rand_like((n, case["width"]), seed + 100).requires_grad_(True)
        s["gy"] = _rand_like((n, case["width"]), seed + 200)
        s["model"] = nn.APPNP(case["hops"], 0.1)
    elif kind == "gat":
        s["csc"] = _attention_graph(case, seed)
        s["x"] = _rand_like((n, case["fin"]), seed + 100)
        torch.manual_seed(seed)
        c = case["heads"] * case["dim"]
        s["layer"] = nn.GATConv(case["fin"], c, case["edges"], heads=case["heads"]).cuda()
        s["gy"] = _rand_like((n, c), seed + 200)
    elif kind == "edge_ops":
        s["csc"] = _attention_graph(case, seed)
        E, c, h = case["edges"], case["channels"], case["heads"]
        s["x"] = _rand_like((n, c), seed + 100).requires_grad_(True)
        s["score"] = _rand_like((E, h), seed + 101).requires_grad_(True)
        s["msg"] = _rand_like((E, c), seed + 102).requires_grad_(True)
        s["g_score"] = _rand_like((E, h), seed + 103)
        s["g_edge"] = _rand_like((E, c), seed + 104)
        s["g_node"] = _rand_like((n, c), seed + 105)
    else:
        scale = max(1, (n - 1).bit_length())
        src, dst = synth.rmat_edges(scale, case["edges"], seed, device="cuda")
        g = torch.Generator(device="cuda").manual_seed(seed + 2)
        perm = torch.randperm(src.numel(), device="cuda", generator=g)
        src, dst = src[perm] % n, dst[perm] % n
        del perm
        # one entry in 65536 is a self-loop, a fixed number, so that the normalised list has a fixed length
        dst = torch.where(src == dst, (dst + 1) % n, dst)
        dst[::65536] = src[::65536]
        s["ei"] = torch.stack([src.to(torch.int32), dst.to(torch.int32)])
        s["w"] = torch.rand(case["edges"], device="cuda", generator=g) + 0.5 if case["weighted"] else None
    return s


# ------------------------------------------------------------------------------ one pass
def _train_step(x, csc, csr, labels, conv1, conv2, rows=None):
    logits = conv2(conv1(x, csc, csr), csc, csr)
    if rows is not None:                         # a sampled batch is trained on its seed nodes
        logits = logits[rows]
    loss = torch.nn.functional.cross_entropy(logits, labels)
    params = [conv1.weight, conv1.bias, conv2.weight, conv2.bias]
    grads = torch.autograd.grad(loss, params)
    return {"logits": logits.detach(), "loss": loss.detach(), "grads": list(grads)}


def run(state):
    s, case = state, state["case"]
    kind = case["kind"]
    if kind == "gcn_step":
        return _train_step(s["x"], s["csc"], s["csr"], s["labels"], s["conv1"], s["conv2"])
    if kind == "gcn_infer":
        with torch.no_grad():
            return s["conv2"](s["conv1"](s["x"], s["csc"], s["csr"]), s["csc"], s["csr"])
    if kind == "minibatch":
        b = sampling.sample_one([case["fan0"], case["fan1"]], s["csc"].column_offset, s["csc"].row_indices, s["seeds"],
                                s["x"], s["labels"], seed=s["seed"])
        rows = torch.searchsorted(b.local2global, s["seeds"])
        return _train_step(b.X, b.csc, b.csr, b.target_lab[rows], s["conv1"], s["conv2"], rows)
    if kind == "spmm":
        y = jg.aggregateWithWeight(s["x"], s["csc"], s["csr"])
        return (y.detach(), torch.autograd.grad(y, s["x"], s["gy"])[0]) if case["backward"] else y
    if kind == "appnp":
        y = s["model"](s["x"], s["csc"], s["csr"])
        return y.detach(), torch.autograd.grad(y, s["x"], s["gy"])[0]
    if kind == "gat":
        if not case["backward"]:
            with torch.no_grad():
                return s["layer"](s["x"], s["csc"])
        y = s["layer"](s["x"], s["csc"])
        return y.detach(), list(torch.autograd.grad(y, [s["layer"].weight, s["layer"].edge_weight], s["gy"]))
    if kind == "edge_ops":
        alpha = ops.EdgeSoftmax(s["score"], s["csc"])
        g_score, = torch.autograd.grad(alpha, s["score"], s["g_score"])
        edge = ops.ScatterToEdge(s["x"], s["csc"], "src")
        g_x, = torch.autograd.grad(edge, s["x"], s["g_edge"])
        node = ops.ScatterToVertex(s["msg"], s["csc"], "src")
        g_msg, = torch.autograd.grad(node, s["msg"], s["g_node"])
        return {"alpha": alpha.detach(), "g_score": g_score, "edge": edge.detach(), "g_x": g_x, "node": node.detach(), "g_msg": g_msg}
    csc, csr = jg.gcn_norm_csc_csr(s["ei"], s["w"], case["nodes"])
    return [csc.row_indices, csc.column_offset, csc.edge_weight, csr.column_indices, csr.row_offset, csr.edge_weight]


# ------------------------------------------------------------------------------ what a pass cannot do without
def _entries(case):
    """Entries of the normalised graph: distinct mirrored edges and one loop per node."""
    if case.get("graph") == "citation":
        return 2 * case["edges"] + case["nodes"]
    return int(2 * case["edges"] * _DISTINCT) + case["nodes"]


def work(case):
    """Bytes: every input read once, every output written once; flops: two per multiply-add."""
    kind, n = case["kind"], case["nodes"]
    if kind in ("gcn_step", "gcn_infer"):
        nnz, f, h, c = _entries(case), case["fin"], case["hidden"], case["classes"]
        one_structure = 8 * nnz + 4 * (n + 1)
        if kind == "gcn_infer":
            return {"bytes": one_structure + 4 * (n * f + f * h + h + h * c + c + n * c), "flops": 2 * n * (f * h + h * c) + 2 * nnz * (h + c)}
        return {"bytes": 2 * one_structure + 8 * n + 4 * (n * f + n * c) + 8 * (f * h + h + h * c + c),
                "flops": 2 * n * (2 * f * h + 3 * h * c) + 4 * nnz * (h + c)}
    if kind == "minibatch":
        nodes = min(n, case["seeds"] * (1 + case["fan0"]) * (1 + case["fan1"]) // 3)
        entries = case["seeds"] * case["fan0"] * (1 + case["fan1"]) // 2
        f, h, c = case["fin"], case["hidden"], case["classes"]
        return {"bytes": 8 * nodes * f + 4 * entries * 6 + 4 * nodes * (c + 6) + 8 * (f * h + h * c),
                "flops": 2 * nodes * (2 * f * h + 3 * h * c) + 4 * entries * (h + c)}
    if kind == "spmm":
        nnz, f = _entries(case), case["width"]
        k = 2 if case["backward"] else 1
        return {"bytes": k * (8 * nnz + 4 * (n + 1) + 8 * n * f), "flops": 2 * k * nnz * f}
    if kind == "appnp":
        nnz, f = _entries(case), case["width"]
        return {"bytes": 2 * (8 * nnz + 4 * (n + 1) + 8 * n * f), "flops": 2 * case["hops"] * (2 * nnz * f + 3 * n * f)}
    if kind == "gat":
        e, f, c, h = case["edges"], case["fin"], case["heads"] * case["dim"], case["heads"]
        if not case["backward"]:
            return {"bytes": 4 * e + 4 * (n + 1) + 4 * (n * f + f * c + 2 * c + n * c), "flops": 2 * n * f * c + e * (4 * c + 4 * h)}
        return {"bytes": 8 * e + 8 * (n + 1) + 4 * (n * f + 2 * n * c) + 8 * (f * c + 2 * c), "flops": 4 * n * f * c + e * (16 * c + 20 * h)}
    if kind == "edge_ops":
        e, c, h = case["edges"], case["channels"], case["heads"]
        return {"bytes": 4 * e * (5 * h + 4 * c) + 16 * n * c + 16 * e, "flops": 2 * e * c + 12 * e * h}
    m = case["edges"] + n
    return {"bytes": (12 if case["weighted"] else 8) * case["edges"] + 16 * m + 8 * (n + 1), "flops": 0}


def tolerance(case):
    """Relative errors another correct implementation at the same precision shows: about four times what each
    kind differs from the same path in float64."""
    kind = case["kind"]
    if kind in ("gcn_step", "minibatch") or (kind == "gat" and case["backward"]):
        # TF32 products in both directions: gradients 0.5 to 1.2 per cent off (ReLU masks flip at zero), single
        # entries of a sparse weight gradient by up to its rms
        return {"rel": 3e-2}
    if kind == "gcn_infer":
        return {"rel": 6e-3, "max": 2e-2}        # two TF32 products: 1.5e-3, single values 5e-3
    if kind == "gat":
        return {"rel": 3.5e-3, "max": 1.2e-2}    # one TF32 product, fp32 attention: 8e-4, single values 3e-3
    return {"rel": 1e-5}                         # fp32 sums: 2e-8 to 1.5e-6; whole numbers are exact


# ------------------------------------------------------------------------------ the same in 64 bits
class _Product64(torch.autograd.Function):
    """``A x`` with the transpose at hand for the backward, both sparse, in float64."""

    @staticmethod
    def forward(ctx, x, a, a_t):
        ctx.a_t = a_t
        return a @ x

    @staticmethod
    def backward(ctx, g):
        return ctx.a_t @ g.contiguous(), None, None


def _sparse64(off, idx, w, n):
    return torch.sparse_csr_tensor(off, idx, w.double(), (n, n), check_invariants=False)


def _gcn64(x, csc, csr, conv1, conv2):
    n = csc.column_offset.numel() - 1
    a = _sparse64(csc.column_offset, csc.row_indices, csc.edge_weight, n)
    a_t = _sparse64(csr.row_offset, csr.column_indices, csr.edge_weight, n)
    params = [p.detach().double().requires_grad_(True) for p in (conv1.weight, conv1.bias, conv2.weight, conv2.bias)]
    hidden = torch.relu(_Product64.apply(x.double() @ params[0], a, a_t) + params[1])
    return _Product64.apply(hidden @ params[2], a, a_t) + params[3], params


def _train_step64(x, csc, csr, labels, conv1, conv2, rows=None):
    logits, params = _gcn64(x, csc, csr, conv1, conv2)
    if rows is not None:
        logits = logits[rows]
    loss = torch.nn.functional.cross_entropy(logits, labels)
    return {"logits": logits.detach(), "loss": loss.detach(), "grads": list(torch.autograd.grad(loss, params))}


def _destinations(off):
    return torch.repeat_interleave(torch.arange(off.numel() - 1, device=off.device), (off[1:] - off[:-1]).long())


def _segment_sum64(v, dst, n):
    return torch.zeros((n,) + v.shape[1:], dtype=torch.float64, device=v.device).index_add_(0, dst, v)


def _segment_softmax64(m, dst, n):
    top = torch.full((n,), -math.inf, dtype=torch.float64, device=m.device).scatter_reduce_(0, dst, m, "amax")
    p = torch.exp(m - top[dst])
    return p / _segment_sum64(p, dst, n)[dst]


def _gat64(case, s):
    """One head at a time; the backward by hand, so that no per-edge rows are kept."""
    n, heads, dim = case["nodes"], case["heads"], case["dim"]
    layer, off, idx = s["layer"], s["csc"].column_offset, s["csc"].row_indices
    x, weight, vec = s["x"].double(), layer.weight.detach().double(), layer.edge_weight.detach().double()[:, 0]
    h = torch.relu(x @ weight)
    c = heads * dim
    dst, src = _destinations(off), idx.long()
    y, g_h, g_vec = torch.empty_like(h), torch.zeros_like(h), torch.zeros_like(vec)
    for k in range(heads):
        cols = slice(k * dim, (k + 1) * dim)
        hk, a_s, a_d = h[:, cols].contiguous(), vec[cols], vec[c + k * dim:c + (k + 1) * dim]
        logit = (hk @ a_s)[src] + (hk @ a_d)[dst]
        alpha = _segment_softmax64(torch.nn.functional.leaky_relu(logit, 0.2), dst, n)
        y[:, cols] = _sparse64(off, idx, alpha, n) @ hk
        if not case["backward"]:
            continue
        g = s["gy"][:, cols].double()
        g_alpha = torch.empty_like(alpha)
        step = 1 << 22
        for e in range(0, alpha.numel(), step):
            g_alpha[e:e + step] = (g[dst[e:e + step]] * hk[src[e:e + step]]).sum(1)
            g_h[:, cols].index_add_(0, src[e:e + step], alpha[e:e + step, None] * g[dst[e:e + step]])
        g_logit = alpha * (g_alpha - _segment_sum64(alpha * g_alpha, dst, n)[dst])
        g_logit = torch.where(logit > 0, g_logit, 0.2 * g_logit)
        by_src, by_dst = _segment_sum64(g_logit, src, n), _segment_sum64(g_logit, dst, n)
        g_h[:, cols] += by_src[:, None] * a_s + by_dst[:, None] * a_d
        g_vec[cols], g_vec[c + k * dim:c + (k + 1) * dim] = by_src @ hk, by_dst @ hk
    if not case["backward"]:
        return y
    return y, [x.t() @ (g_h * (h > 0)), g_vec[:, None]]


def _edge_ops64(case, s):
    n = case["nodes"]
    dst, src = _destinations(s["csc"].column_offset), s["csc"].row_indices.long()
    alpha, g_score = [], []
    for k in range(case["heads"]):
        a, g = _segment_softmax64(s["score"].detach()[:, k].double(), dst, n), s["g_score"][:, k].double()
        alpha.append(a)
        g_score.append(a * (g - _segment_sum64(a * g, dst, n)[dst]))
    return {"alpha": torch.stack(alpha, 1), "g_score": torch.stack(g_score, 1), "edge": s["x"].detach().double()[src],
            "g_x": _segment_sum64(s["g_edge"].double(), src, n), "node": _segment_sum64(s["msg"].detach().double(), dst, n),
            "g_msg": s["g_node"].double()[dst]}


def _convert64(case, s):
    """The weights; the whole numbers beside them are compared as they are."""
    n = case["nodes"]
    src, dst = s["ei"]
    w = torch.ones(src.numel(), device="cuda") if s["w"] is None else s["w"]
    loop_w = torch.ones(n, device="cuda")
    loops = torch.nonzero(src == dst)[:, 0]                       # a node's last loop entry gives its weight
    at = torch.full((n,), -1, device="cuda").scatter_reduce_(0, src[loops].long(), loops, "amax")
    loop_w = torch.where(at >= 0, w[at.clamp(min=0)], loop_w)
    ids = torch.arange(n, dtype=torch.int32, device="cuda")
    keep = src != dst
    src, dst, w = torch.cat([src[keep], ids]), torch.cat([dst[keep], ids]), torch.cat([w[keep], loop_w]).double()
    inv = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, dst, w).rsqrt()
    w = inv[src] * w * inv[dst]
    return [None, None, w[torch.sort(dst, stable=True)[1]], None, None, w[torch.sort(src, stable=True)[1]]]


def exact(case, seed):
    """What ``run`` returns, from plain torch in float64 on the structure that the inputs hold.  A sampled
    batch is whole numbers: the exact values are those of the step on that batch."""
    s = prepare(case, seed)
    kind = case["kind"]
    if kind == "gcn_step":
        return _train_step64(s["x"], s["csc"], s["csr"], s["labels"], s["conv1"], s["conv2"])
    if kind == "gcn_infer":
        with torch.no_grad():
            return _gcn64(s["x"], s["csc"], s["csr"], s["conv1"], s["conv2"])[0]
    if kind == "minibatch":
        b = sampling.sample_one([case["fan0"], case["fan1"]], s["csc"].column_offset, s["csc"].row_indices, s["seeds"], seed=s["seed"])
        nodes = b.local2global.long()
        rows = torch.searchsorted(b.local2global, s["seeds"])
        return _train_step64(s["x"][nodes], b.csc, b.csr, s["labels"][nodes][rows], s["conv1"], s["conv2"], rows)
    if kind in ("spmm", "appnp"):
        n, x = case["nodes"], s["x"].detach().double()
        a = _sparse64(s["csc"].column_offset, s["csc"].row_indices, s["csc"].edge_weight, n)
        if kind == "spmm" and not case["backward"]:
            return a @ x
        a_t = _sparse64(s["csr"].row_offset, s["csr"].column_indices, s["csr"].edge_weight, n)
        g = s["gy"].double()
        if kind == "spmm":
            return a @ x, a_t @ g
        y, gx = x, torch.zeros_like(g)
        for _ in range(case["hops"]):
            y = 0.1 * x + 0.9 * (a @ y)
            gx = gx + 0.1 * g
            g = 0.9 * (a_t @ g)
        return y, gx + g
    if kind == "gat":
        with torch.no_grad():
            return _gat64(case, s)
    if kind == "edge_ops":
        with torch.no_grad():
            return _edge_ops64(case, s)
    return _convert64(case, s)
