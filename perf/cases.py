"""The work that users of this framework have it do, as cases that can be timed.

Six kinds, all through the public entry points:

  train   one training step of a stacked GCN: zero_grad, forward, fused loss, backward, fused optimizer step;
          issued eagerly or replayed as one CUDA graph
  eval    the script's test(): forward without autograd, argmax, hits per split
  layer   one GCNConv (bias, ReLU), forward only or forward and backward, on a CSR or a dense adjacency
  matmul  one dense product: the reference's operator names, or gemm() with a layout and a precision
  spmm    one spmm_cusparse() call on a torch sparse tensor
  build   edge list -> normalised CSR adjacency

The listed sizes are the configurations this library is benchmarked on (graphcuda_b200/synth.py) and the shapes of
its tests; draw() spreads over the ranges around them.  Graphs are seeded R-MAT or preferential-attachment graphs,
features normal or bag-of-words, labels uniform: the distributions of the same configurations.
"""
import math

import torch

import graphcuda_b200 as gc
from graphcuda_b200 import synth
from graphcuda_b200.models import GCN

DEV = "cuda"


# ------------------------------------------------------------------ cases
def listed():
    cora = dict(graph="pref", nodes=2708, edges=5429, dims="1433-16-7", precision="fp32")
    arxiv = dict(graph="rmat", nodes=169_343, edges=1_166_243)
    return [
        # The reference's own script: 2 layers on a Cora-sized graph, SGD.  Launches and host work dominate.
        dict(name="train_cora_eager", kind="train", optimizer="sgd", replay=False, split=True, **cora),
        # The same epoch as most users of a small graph should run it: Adam, recorded once, replayed.
        dict(name="train_cora_replay", kind="train", optimizer="adam", replay=True, split=True, **cora),
        # The script's test(), called after every epoch.
        dict(name="eval_cora", kind="eval", **cora),
        # A single layer of a deeper model at citation-graph size: forward and both gradients.
        dict(name="layer_arxiv", kind="layer", adjacency="csr", dims="128-256", precision="fp32", backward=True, **arxiv),
        # A 3-layer model at the same size in the reduced-precision tier.
        dict(name="train_arxiv_bf16", kind="train", optimizer="adam", replay=False, split=False, dims="128-256-256-47",
             precision="bf16", **arxiv),
        # The largest configuration, full batch: the headline benchmark.
        dict(name="train_products", kind="train", optimizer="adam", replay=False, split=False, dims="100-256-256-47",
             precision="fp32", graph="rmat", nodes=2_449_029, edges=61_859_140),
        # The README's calling convention: a dense adjacency.  Inference in fp32 ...
        dict(name="layer_dense_fp32", kind="layer", adjacency="dense", graph="er", nodes=32_768, edges=5_368_545,
             dims="512-256", precision="fp32", backward=False),
        # ... and a training step of that layer in the bf16 tier.
        dict(name="layer_dense_bf16", kind="layer", adjacency="dense", graph="er", nodes=32_768, edges=5_368_545,
             dims="512-256", precision="bf16", backward=True),
        # The operator sweep of the reference's matmul tests: a square ...
        dict(name="matmul_4096", kind="matmul", op="matmul4", m=4096, n=4096, k=4096, layout="nn", precision="fp32"),
        # ... and ragged sizes with unaligned row pitches.
        dict(name="matmul_ragged", kind="matmul", op="gemm_cublas", m=2049, n=515, k=1433, layout="nn",
             precision="fp32"),
        # The stand-alone aggregation operator on a COO tensor with an odd feature width (the class count).
        dict(name="spmm_coo_odd", kind="spmm", layout="coo", width=47, **arxiv),
        # Preprocessing: what a user pays once per graph, or per batch when graphs are sampled.
        dict(name="build_arxiv", kind="build", reorder=False, **arxiv),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _drawn_graph(rng, most=600_000):
    nodes = _log(rng, 1000, most)
    return dict(graph="rmat", nodes=nodes, edges=int(nodes * math.exp(rng.uniform(math.log(2.0), math.log(25.0)))))


def _aligned(case):
    """TF32 reads its operands in place and takes 16-byte row pitches only: sizes in multiples of 8."""
    if case.get("precision") == "tf32":
        up = lambda x: (x + 7) // 8 * 8  # noqa: E731
        case.update({k: up(case[k]) for k in ("m", "n", "k") if k in case})
        if "dims" in case:
            case["dims"] = "-".join(str(up(int(d))) for d in case["dims"].split("-"))
        if case.get("adjacency") == "dense":
            case["nodes"] = up(case["nodes"])
    return case


def draw(rng):
    return _aligned(_draw(rng))


def _draw(rng):
    kind = rng.choices(("train", "eval", "layer", "matmul", "spmm", "build"), (6, 2, 5, 4, 2, 1))[0]
    if kind == "matmul":
        op = rng.choice(("matmul1", "matmul2", "matmul3", "matmul4", "gemm_cublas", "gemm", "gemm", "gemm"))
        layout = rng.choice(("nn", "nn", "tn", "nt")) if op == "gemm" else "nn"
        precision = rng.choice(("fp32", "fp32", "tf32", "bf16")) if op == "gemm" else "fp32"
        if rng.random() < 0.3:  # feature transforms: tall and narrow
            m, n, k = _log(rng, 20_000, 1_200_000), _log(rng, 7, 256), _log(rng, 16, 512)
        else:
            m, n, k = (_log(rng, 64, 6000) for _ in range(3))
        if layout == "tn" and rng.random() < 0.5:  # weight gradients: a long sum
            m, n, k = _log(rng, 16, 512), _log(rng, 7, 256), _log(rng, 2000, 600_000)
        if rng.random() < 0.5:  # half of them at sizes that users choose, half as they fall
            m, n, k = (max(8, (x + 7) // 8 * 8) for x in (m, n, k))
        return dict(kind=kind, op=op, m=m, n=n, k=k, layout=layout, precision=precision)
    if kind == "build":
        return dict(kind=kind, reorder=rng.random() < 0.3, **_drawn_graph(rng))
    if kind == "spmm":
        return dict(kind=kind, layout=rng.choice(("coo", "csr")), width=_log(rng, 5, 512), **_drawn_graph(rng))
    if kind == "layer" and rng.random() < 0.3:
        nodes = _log(rng, 1000, 20_000)
        return dict(kind=kind, adjacency="dense", graph="rmat", nodes=nodes, edges=nodes * rng.randint(2, 20),
                    dims="%d-%d" % (_log(rng, 16, 512), _log(rng, 7, 256)),
                    precision=rng.choice(("fp32", "fp32", "tf32", "bf16")), backward=rng.random() < 0.6)
    g = _drawn_graph(rng)
    wide = 1433 if g["nodes"] < 20_000 else 512 if g["nodes"] < 200_000 else 256
    feat, hidden, classes = _log(rng, 16, wide), rng.choice((16, 32, 64, 128, 256, _log(rng, 16, 256))), rng.randint(2, 64)
    if kind == "layer":
        return dict(kind=kind, adjacency="csr", dims="%d-%d" % (feat, rng.choice((hidden, classes))),
                    precision=rng.choice(("fp32", "fp32", "fp32", "tf32", "bf16")), backward=rng.random() < 0.7, **g)
    # Replayed steps are left to the listed case: recording is for graphs of that size.
    dims = "-".join(str(d) for d in [feat] + [hidden] * rng.randint(1, 2) + [classes])
    if kind == "eval":
        return dict(kind=kind, dims=dims, precision="fp32", **g)
    return dict(kind=kind, dims=dims, precision=rng.choice(("fp32", "fp32", "fp32", "tf32", "bf16")),
                optimizer=rng.choice(("sgd", "adam")), replay=False, split=rng.random() < 0.3, **g)


# ------------------------------------------------------------------ inputs
def _edge_index(case, seed):
    """Directed edge list (both directions of every edge), int64 on the GPU."""
    n, e = case["nodes"], case["edges"]
    if case["graph"] == "pref":
        edges = synth.preferential_attachment_edges(n, e, seed).to(DEV)
    elif case["graph"] == "er":
        edges = synth.erdos_renyi_edges(n, 2.0 * e / (n * (n - 1.0)), seed, device=DEV)
    else:
        edges = synth.rmat_edges((n - 1).bit_length(), n, e, seed, device=DEV)
    return synth.symmetrize(edges)


def _adjacency(case, seed):
    return gc.normalized_adjacency(_edge_index(case, seed), case["nodes"], symmetric=True)


def _dims(case):
    return [int(d) for d in case["dims"].split("-")]


def _features(case, width, seed):
    if case["graph"] == "pref":
        return synth.bow_features(case["nodes"], width, 0.0127, seed, device=DEV)
    return synth.normal_features(case["nodes"], width, seed, device=DEV)


def _optimizer(case, model, seed):
    if case["optimizer"] == "sgd":
        return gc.FusedSGD(model.parameters(), lr=1.0)
    opt = gc.FusedAdam(model.parameters(), lr=0.01)
    # A run in progress: moments of earlier steps, about the size of the gradients.  (From zero moments the first
    # update is lr * sign(gradient), which the last bit of a gradient near zero decides.)
    g = torch.Generator(device=DEV).manual_seed(seed + 3)
    for p in model.parameters():
        opt.state[p]["exp_avg"] = 1e-3 * torch.randn(p.shape, generator=g, device=DEV)
        opt.state[p]["exp_avg_sq"] = 1e-6 * (0.5 + torch.rand(p.shape, generator=g, device=DEV))
    return opt


def _uniform(rows, cols, gen, transposed):
    """rows x cols, uniform(-1, 1); transposed: a view of a cols x rows matrix."""
    shape = (cols, rows) if transposed else (rows, cols)
    t = torch.rand(shape, generator=gen, device=DEV) * 2 - 1
    return t.t() if transposed else t


def prepare(case, seed):
    kind = case["kind"]
    if kind == "matmul":
        gen = torch.Generator(device=DEV).manual_seed(seed)
        return dict(case=case, A=_uniform(case["m"], case["k"], gen, case["layout"][0] == "t"),
                    B=_uniform(case["k"], case["n"], gen, case["layout"][1] == "t"))
    if kind == "build":
        return dict(case=case, edge_index=_edge_index(case, seed))
    adj = _adjacency(case, seed)
    if kind == "spmm":
        A = adj.to_sparse_coo()
        if case["layout"] == "csr":
            A = A.to_sparse_csr()
        return dict(case=case, A=A, B=synth.normal_features(case["nodes"], case["width"], seed + 1, device=DEV))
    dims = _dims(case)
    torch.manual_seed(seed + 2)  # the modules initialise their weights from the global generator
    if kind == "layer":
        conv = gc.GCNConv(dims[0], dims[1], apply_relu=True, bias=True, precision=case["precision"]).to(DEV)
        x = _features(case, dims[0], seed + 1)
        if case["adjacency"] == "dense":
            adj = adj.to_sparse_coo().to_dense()
        if not case["backward"]:
            return dict(case=case, conv=conv, adj=adj, x=x)
        return dict(case=case, conv=conv, adj=adj, x=x.requires_grad_(),
                    dy=synth.normal_features(case["nodes"], dims[1], seed + 4, device=DEV))
    model = GCN(dims, precision=case["precision"]).to(DEV)
    s = dict(case=case, model=model, adj=adj, x=_features(case, dims[0], seed + 1),
             y=synth.uniform_labels(case["nodes"], dims[-1], seed + 5, device=DEV))
    n = case["nodes"]
    few = (140, 500, 1000) if n >= 1640 else (n // 10, n // 4, n // 3)
    if kind == "eval":
        s["masks"] = [m.to(DEV) for m in synth.planetoid_split(n, *few)]
        return s
    s["mask"] = synth.planetoid_split(n, *few)[0].to(DEV) if case["split"] else None
    s["scale"] = 1.0 / (few[0] if case["split"] else n)
    s["opt"] = _optimizer(case, model, seed)
    if case["replay"]:
        s["step"] = gc.GraphedTrainStep(model, adj, s["x"], s["y"], s["opt"], row_mask=s["mask"])
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "matmul":
        if case["op"] == "gemm":
            return gc.gemm(s["A"], s["B"], precision=case["precision"])
        return getattr(gc, case["op"])(s["A"], s["B"])
    if kind == "spmm":
        return gc.spmm_cusparse(s["A"], s["B"])
    if kind == "build":
        adj = gc.normalized_adjacency(s["edge_index"], case["nodes"], reorder="degree" if case["reorder"] else None)
        return [adj.rowptr, adj.col, adj.val] + ([adj.perm, adj.inv_perm] if case["reorder"] else [])
    if kind == "layer":
        conv, x = s["conv"], s["x"]
        if not case["backward"]:
            with torch.no_grad():
                return conv(x, s["adj"])
        x.grad = conv.weights.grad = conv.bias.grad = None
        y = conv(x, s["adj"])
        y.backward(s["dy"])
        return [y.detach(), x.grad, conv.weights.grad, conv.bias.grad]
    if kind == "eval":
        return list(s["model"].evaluate(s["x"], s["adj"], s["y"], s["masks"]))
    opt, params = s["opt"], list(s["model"].parameters())
    if case["replay"]:
        loss = s["step"].step()
    else:
        opt.zero_grad(set_to_none=True)
        out = s["model"](s["x"], s["adj"], log_softmax=False)
        loss = gc.log_softmax_nll_loss(out, s["y"], s["mask"], scale=s["scale"])
        loss.backward()
        opt.step()
    state = [opt.state[p][k] for p in params for k in ("exp_avg", "exp_avg_sq")] if case["optimizer"] == "adam" else []
    return [loss.detach()] + [p.grad for p in params] + [p.detach() for p in params] + state


# ------------------------------------------------------------------ what a pass cannot do without
def _layers_work(n, nnz_flops, dims, backward, dx_first):
    """Flops of a stack of layers: each product once, aggregations on the narrower side."""
    flops = 0.0
    for i, (a, b) in enumerate(zip(dims[:-1], dims[1:])):
        flops += 2.0 * n * a * b + nnz_flops * min(a, b)
        if backward:
            need_dx = i > 0 or dx_first
            flops += 2.0 * n * a * b * (2 if need_dx else 1)
            flops += nnz_flops * min(a, b) if need_dx or b < a else 0.0
    return flops


def work(case):
    kind = case["kind"]
    if kind == "matmul":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 4.0 * (m * k + k * n + m * n), "flops": 2.0 * m * n * k}
    n, e = case["nodes"], case["edges"]
    nnz = 2 * e + n
    if kind == "build":
        return {"bytes": 16.0 * 2 * e + 4.0 * (n + 1) + 8.0 * nnz + (16.0 * n if case["reorder"] else 0.0), "flops": 0.0}
    dense = case.get("adjacency") == "dense"
    adj_bytes = 4.0 * n * n if dense else 4.0 * (n + 1) + 8.0 * nnz
    nnz_flops = 2.0 * n * n if dense else 2.0 * nnz
    if kind == "spmm":
        w = case["width"]
        return {"bytes": 4.0 * (n + 1) + (8.0 if case["layout"] == "csr" else 12.0) * nnz + 8.0 * n * w,
                "flops": nnz_flops * w}
    dims = _dims(case)
    weights = sum(a * b for a, b in zip(dims[:-1], dims[1:]))
    bytes_ = adj_bytes + 4.0 * n * dims[0] + 4.0 * weights
    if kind == "layer":
        if case["backward"]:  # dY in, Y and dX out, dW out
            return {"bytes": bytes_ + 4.0 * n * (2 * dims[1] + dims[0]) + 4.0 * weights,
                    "flops": _layers_work(n, nnz_flops, dims, True, True)}
        return {"bytes": bytes_ + 4.0 * n * dims[1], "flops": _layers_work(n, nnz_flops, dims, False, False)}
    if kind == "eval":
        return {"bytes": bytes_ + 8.0 * n + 3.0 * n + 8.0 * n, "flops": _layers_work(n, nnz_flops, dims, False, False)}
    per_weight = 2 + (4 if case["optimizer"] == "adam" else 0)  # gradient and weight out; moments in and out
    return {"bytes": bytes_ + 8.0 * n + 4.0 * weights * per_weight,
            "flops": _layers_work(n, nnz_flops, dims, True, False)}


def tolerance(case):
    kind = case["kind"]
    if kind == "build":
        return "exact"
    if kind == "eval":
        return {"rel": 0.0, "differ": 1e-3}  # argmax between classes that differ in the last bits
    if case.get("precision", "fp32") != "fp32":
        return {"rel": 2e-2, "max": 0.9}
    if kind == "spmm":
        return {"rel": 1e-5}
    if kind == "matmul":
        # fp32 operands as three tensor-core products: the sums are truncated, so the error grows with their length
        return {"rel": 2e-5 if case["k"] <= 1024 else 1e-4, "max": 1e-3}
    if kind == "layer" and not case["backward"]:
        return {"rel": 2e-5 if case["adjacency"] == "csr" else 1e-4, "max": 1e-3}
    # Gradients behind a ReLU: an activation within rounding (1e-6) of zero may fall on either side, so a share of
    # about 1e-6 of the gated gradient's entries may be there or not -- 1e-3 of its norm.
    return {"rel": 3e-3, "max": 0.9}
