"""Timed cases of the CBM products, through the calls a user's program makes.

Every case builds its graph, its operator and its operands from a seed:

* ``community``  nodes in communities of 64, most links inside the community
  (the 4,096-node graph; with ``graphs`` > 1 a batch of such graphs, sizes
  spread log-uniformly, mean degrees over 8 to 40);
* ``powerlaw``   Chung-Lu degrees, then a share of the rows replaced by flipped
  copies of other rows, which is what the compression tree is made of.

The laws are those of ``cbm.synthetic``; they are restated here on the GPU so
that a million-node graph takes milliseconds.  ``call`` names the public entry
point:

* ``AX`` / ``ADX`` / ``DADX``  ``cbm4mm`` / ``cbm4ad`` / ``cbm4dad`` ``.matmul(x, y)``,
  or ``cbm_batch(...).matmul`` with several graphs;
* ``ADX_T``    ``cbm4ad.adjoint(g, dx)``: the backward of A D^-1/2 (not self-adjoint);
* ``GIN``      ``cbm4mm.matmul_add(x, y, epsilon)``;
* ``OP_DADX``  ``cbm_mkl_cpp.s_spmm_fused_update_csr_int32`` on CUDA tensors: the
  stateless operator with the caller's own CSR and tree arrays;
* ``GCN``      one training step (forward, loss, backward) of ``cbm.gcn.GCN``.
"""
import math
import os
import random  # noqa: F401  (draw() takes a random.Random)
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cbm-gpu_b200"))

BF16, F32 = "bfloat16", "float32"
EPSILON = 0.25  # the GIN form's epsilon
HIDDEN, CLASSES = 256, 40  # the GCN's widths after its input


def _powerlaw(name, call, n, cols, x, y, mean, exponent, dup, flip, alpha):
    return dict(name=name, call=call, graph="powerlaw", graphs=1, n=n, cols=cols, x=x, y=y, mean=mean,
                exponent=exponent, dup=dup, flip=flip, alpha=alpha)


def _community(name, call, n, cols, x, y, mean, graphs=1):
    return dict(name=name, call=call, graph="community", graphs=graphs, n=n, cols=cols, x=x, y=y, mean=mean,
                exponent=0.0, dup=0.0, flip=0.0, alpha=0)


def listed():
    gcn = dict(mean=14.0, exponent=2.1, dup=0.25, flip=0.10, alpha=0)  # the GCN graph's law: a deep tree
    head = dict(mean=20.0, exponent=2.1, dup=0.30, flip=0.10, alpha=8)  # the 1M-node graph's law
    return [
        # a small graph that is multiplied again and again: launch and latency
        _community("small-ax-64", "AX", 4096, 64, F32, F32, 32.0),
        # the aggregations of a two-layer GCN in BF16: its input width, then
        # its class width with FP32 logits
        _powerlaw("gcn-dadx-128-bf16", "DADX", 170_000, 128, BF16, BF16, **gcn),
        _powerlaw("gcn-dadx-40-bf16", "DADX", 170_000, 40, BF16, F32, **gcn),
        # the same graph in plain FP32
        _powerlaw("gcn-dadx-128-f32", "DADX", 170_000, 128, F32, F32, **gcn),
        # an odd class count: rows that no 16-byte vector divides
        _powerlaw("odd-dadx-47-f32", "DADX", 99_991, 47, F32, F32, **gcn),
        # the GIN aggregation A X + (1 + eps) X
        _powerlaw("gin-64-f32", "GIN", 100_000, 64, F32, F32, **gcn),
        # backward of an operator that is not its own transpose
        _powerlaw("adjoint-adx-40-f32", "ADX_T", 170_000, 40, F32, F32, **gcn),
        # X and Y far larger than L2: the million-node product
        _powerlaw("large-dadx-256-f32", "DADX", 1_000_000, 256, F32, F32, **head),
        # long rows, X stored in BF16, FP32 results
        _powerlaw("dense-adx-128-bf16", "ADX", 400_000, 128, BF16, F32, 50.0, 2.3, 0.40, 0.05, 16),
        # many graphs in one launch
        _community("batch-dadx-64-bf16", "DADX", 800_000, 64, BF16, F32, 24.0, graphs=48),
        # the stateless operator: the caller's arrays as they are
        _powerlaw("operator-dadx-256-f32", "OP_DADX", 250_000, 256, F32, F32, **head),
        # a whole training step; returns logits and weight gradients
        _powerlaw("gcn-step-bf16", "GCN", 170_000, 128, BF16, F32, **gcn),
    ]


def draw(rng):
    """One more case of the ranges above: sizes over their logarithm, any width
    from one column to 256 (about half of them no multiple of a vector)."""
    call = rng.choice(["AX", "ADX", "DADX", "DADX", "DADX", "GIN", "ADX_T", "OP_DADX", "GCN"])
    n = int(round(math.exp(rng.uniform(math.log(2_000), math.log(200_000)))))
    cols = rng.choice([8, 16, 32, 40, 64, 96, 128, 256]) if rng.random() < 0.5 else \
        int(round(math.exp(rng.uniform(0.0, math.log(256)))))
    x = rng.choice([F32, BF16]) if call in ("AX", "ADX", "DADX", "GIN") else F32
    y = rng.choice([F32, BF16]) if x == BF16 else F32
    if call == "GCN":
        cols, x = rng.choice([32, 64, 100, 128]), rng.choice([F32, BF16])
    if call in ("AX", "ADX", "DADX", "GIN") and rng.random() < 0.35:
        c = _community("", call, n, cols, x, y, float(rng.choice([8, 16, 24, 32, 40])))
        if call != "GIN" and n > 20_000 and rng.random() < 0.6:
            c.update(graphs=rng.randint(2, 16), mean=24.0)
    else:
        alpha = rng.choice([0, 0, 8, 16])
        c = _powerlaw("", call, n, cols, x, y, rng.choice([10.0, 14.0, 20.0, 30.0]),
                      round(rng.uniform(2.1, 2.5), 2), round(rng.uniform(0.1, 0.4), 2), rng.choice([0.05, 0.10]), alpha)
    del c["name"]
    return c


# ---- graphs (on the GPU, from a generator) ---------------------------------------


def _coalesce(r, c, n):
    """Sorted distinct keys r * n + c of the symmetrised edges, no self-loops."""
    keep = r != c
    r, c = r[keep], c[keep]
    return torch.unique(torch.cat([r * n + c, c * n + r]))


def _community_keys(n, mean, g):
    size = 64
    half = max(1, int(round(mean / 2)))
    k_in = min(max(1, int(round(0.75 * half))), size - 1)
    k_out = max(0, half - k_in)
    node = torch.arange(n, device="cuda")
    start = node // size * size
    width = torch.clamp(start + size, max=n) - start
    key = torch.rand(n, size, generator=g, device="cuda")
    other = torch.arange(size, device="cuda")[None, :]
    key[(other >= width[:, None]) | (other == (node - start)[:, None])] = 2.0
    val, pick = torch.topk(key, k_in, dim=1, largest=False)
    ok = val < 1.5
    r = [node[:, None].expand_as(pick)[ok]]
    c = [(start[:, None] + pick)[ok]]
    if k_out:
        r.append(node.repeat_interleave(k_out))
        c.append(torch.randint(0, n, (n * k_out,), generator=g, device="cuda"))
    # the last node always has a link, so that the graph has n nodes
    r.append(node[-1:])
    c.append(node[:1])
    return _coalesce(torch.cat(r), torch.cat(c), n)


def _powerlaw_keys(n, exponent, mean, dup, flip, g):
    w = torch.arange(1, n + 1, dtype=torch.float64, device="cuda") ** (-1.0 / (exponent - 1.0))
    w *= mean / w.mean()
    w = torch.clamp(w, max=math.sqrt(float(w.sum())))
    m = int(round(float(w.sum()) / 2))
    cdf = torch.cumsum(w / w.sum(), 0)
    cdf[-1] = 1.0
    uv = torch.searchsorted(cdf, torch.rand(2, m, generator=g, device="cuda", dtype=torch.float64), right=True)
    uv = torch.randperm(n, generator=g, device="cuda")[torch.clamp(uv, max=n - 1)]
    keys = _coalesce(uv[0], uv[1], n)
    rows, cols = keys // n, keys % n
    ptr = torch.searchsorted(keys, torch.arange(n + 1, device="cuda") * n)
    # a share of the rows become copies of other rows, some entries replaced
    n_copy = int(round(dup * n))
    perm = torch.randperm(n, generator=g, device="cuda")
    copies, pool = perm[:n_copy], perm[n_copy:]
    templ = pool[torch.randint(0, pool.numel(), (n_copy,), generator=g, device="cuda")]
    is_copy = torch.zeros(n, dtype=torch.bool, device="cuda")
    is_copy[copies] = True
    keep = ~is_copy[rows]
    lens = ptr[templ + 1] - ptr[templ]
    owner = torch.repeat_interleave(torch.arange(n_copy, device="cuda"), lens)
    first = torch.cumsum(lens, 0) - lens
    at = ptr[templ][owner] + torch.arange(owner.numel(), device="cuda") - first[owner]
    c_cols = cols[at]
    drop = torch.rand(owner.numel(), generator=g, device="cuda") < flip
    c_cols[drop] = torch.randint(0, n, (int(drop.sum()),), generator=g, device="cuda")
    last = torch.tensor([n - 1], device="cuda")
    return _coalesce(torch.cat([rows[keep], copies[owner], last]), torch.cat([cols[keep], c_cols, last * 0]), n)


def _sizes(case):
    """Node counts and mean degrees of a case's graphs."""
    k = case["graphs"]
    if k == 1:
        return [case["n"]], [case["mean"]]
    # log-spaced over a factor of 64, scaled to the case's total
    s = np.exp(np.linspace(0.0, math.log(64.0), k))
    s = np.maximum(64, np.round(s * case["n"] / s.sum())).astype(int)
    s[-1] += case["n"] - int(s.sum())
    return [int(v) for v in s], [8.0 + 32.0 * ((7 * i) % k) / max(1, k - 1) for i in range(k)]


def _graphs(case, seed):
    """[(keys r * n + c, n)] of the case's graphs."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    out = []
    for n, mean in zip(*_sizes(case)):
        if case["graph"] == "community":
            out.append((_community_keys(n, mean, g), n))
        else:
            out.append((_powerlaw_keys(n, case["exponent"], mean, case["dup"], case["flip"], g), n))
    return out


def _edges(keys, n):
    return torch.stack([keys // n, keys % n]).to(torch.int32).cpu()


def _features(case, seed):
    """The dense operands: features (or a gradient), normally distributed; for
    a GCN also labels."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) + (1 << 32))
    x = torch.randn(case["n"], case["cols"], generator=g, device="cuda").to(getattr(torch, case["x"]))
    labels = torch.randint(0, CLASSES, (case["n"],), generator=g, device="cuda") if case["call"] == "GCN" else None
    return x, labels


# ---- the measured calls -------------------------------------------------------


def prepare(case, seed):
    from cbm import cbm_mkl_cpp
    from cbm.batch import cbm_batch
    from cbm.cbm4ad import cbm4ad
    from cbm.cbm4dad import cbm4dad
    from cbm.cbm4mm import cbm4mm
    from cbm.gcn import GCN

    call = case["call"]
    graphs = _graphs(case, seed)
    if case["graphs"] > 1:
        op = cbm_batch([(_edges(k, n).numpy(), n) for k, n in graphs], alpha=case["alpha"], op=call.lower())
    else:
        ei = _edges(*graphs[0])
        cls = {"AX": cbm4mm, "GIN": cbm4mm, "ADX": cbm4ad, "ADX_T": cbm4ad}.get(call, cbm4dad)
        op = cls(ei, torch.ones(ei.shape[1]), alpha=case["alpha"])
    del graphs
    x, labels = _features(case, seed)
    s = {"call": call, "op": op, "x": x}
    if call == "GCN":
        s["model"] = GCN(op, case["cols"], HIDDEN, CLASSES, act_dtype=x.dtype, seed=int(seed) % (1 << 31))
        s["labels"] = labels
        return s
    s["y"] = torch.empty(case["n"], case["cols"], dtype=getattr(torch, case["y"]), device="cuda")
    if call == "ADX_T":
        op.plan.prepare_adjoint()
    elif call == "OP_DADX":
        crow = op.deltas.crow_indices()
        s["args"] = (crow[:-1].contiguous(), crow[1:].contiguous(), op.deltas.col_indices(), op.deltas.values(), x,
                     op.mca_offset, op.mca_src_idx, op.mca_dst_idx, op.D, s["y"])
        s["operator"] = cbm_mkl_cpp.s_spmm_fused_update_csr_int32
    return s


def run(s):
    call = s["call"]
    if call == "GCN":
        from cbm.gcn import cross_entropy

        m = s["model"]
        m.zero_grad(set_to_none=True)
        logits = m(s["x"])
        cross_entropy(logits, s["labels"]).backward()
        return {"logits": logits.detach(), "w1": m.w1.grad, "w2": m.w2.grad}
    if call == "OP_DADX":
        s["operator"](*s["args"])
    elif call == "ADX_T":
        s["op"].adjoint(s["x"], s["y"])
    elif call == "GIN":
        s["op"].matmul_add(s["x"], s["y"], EPSILON)
    else:
        s["op"].matmul(s["x"], s["y"])
    return s["y"]


def work(case):
    """X read once, Y written once, 4 bytes for each nonzero of A (and D where
    the product scales); two operations per nonzero and column."""
    n, c = case["n"], case["cols"]
    sx, sy = (2 if case[k] == BF16 else 4 for k in ("x", "y"))
    nnz = sum(a * b for a, b in zip(*_sizes(case)))
    if case["call"] == "GCN":
        w = c * HIDDEN + HIDDEN * CLASSES
        # the input, the logits, three products with A, the dense products and their gradients
        return {"bytes": n * c * sx + n * CLASSES * 4 + 3 * nnz * 4,
                "flops": 2 * nnz * (c + 2 * CLASSES) + 2 * n * (2 * c * HIDDEN + 3 * HIDDEN * CLASSES) + w}
    scaled = case["call"] not in ("AX", "GIN")
    return {"bytes": n * c * (sx + sy) + 4 * nnz + (4 * n if scaled else 0), "flops": 2 * nnz * c}


# ---- the same results in 64 bits, by torch alone ----------------------------------


def _matrix(case, seed):
    """The case's A as one sparse CSR matrix of ones (block-diagonal for a batch)."""
    n, rows, cols, off = case["n"], [], [], 0
    for keys, k in _graphs(case, seed):
        rows.append(keys // k + off)
        cols.append(keys % k + off)
        off += k
    r, c = torch.cat(rows), torch.cat(cols)
    ptr = torch.searchsorted(r, torch.arange(n + 1, device="cuda"))
    one = torch.ones(c.numel(), dtype=torch.float64, device="cuda")
    return torch.sparse_csr_tensor(ptr, c, one, (n, n))


def _exact_gcn(case, seed, ahat):
    # the model's initial weights: uniform in +-sqrt(6 / (fan in + fan out))
    g = torch.Generator(device="cpu").manual_seed(int(seed) % (1 << 31))
    w = []
    for shape in ((case["cols"], HIDDEN), (HIDDEN, CLASSES)):
        bound = math.sqrt(6.0 / sum(shape))
        w.append((torch.rand(*shape, generator=g) * (2 * bound) - bound).cuda().double().requires_grad_())
    w1, w2 = w
    x, labels = _features(case, seed)
    ax = ahat(x.double())
    h = torch.relu(ax @ w1)
    hw = h @ w2
    logits = ahat(hw.detach()).requires_grad_()
    torch.nn.functional.cross_entropy(logits, labels).backward()
    hw.backward(ahat(logits.grad))  # D^-1/2 A D^-1/2 of a symmetric A is its own transpose
    return {"logits": logits.detach(), "w1": w1.grad, "w2": w2.grad}


def exact(case, seed):
    call = case["call"]
    a = _matrix(case, seed)
    ptr = a.crow_indices()
    deg = (ptr[1:] - ptr[:-1]).double()[:, None]
    d = torch.where(deg > 0, deg.clamp(min=1.0) ** -0.5, torch.zeros_like(deg))
    if call == "GCN":
        return _exact_gcn(case, seed, lambda v: d * (a @ (d * v)))
    x = _features(case, seed)[0].double()
    if call == "AX":
        return a @ x
    if call == "GIN":
        return a @ x + (1.0 + EPSILON) * x
    if call == "ADX":
        return a @ (d * x)
    if call == "ADX_T":
        return d * (a @ x)  # A is symmetric
    return d * (a @ (d * x))
