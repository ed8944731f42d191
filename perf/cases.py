"""The workloads this library's speed is judged by: what a mixture-of-experts program
has it do, through its public entry points, from the smallest call to the largest.

Every case is a dict of plain values:

  op       "gmm"     one grouped product (``grouped_gemm.ops.gmm``)
           "gather"  the same with the sort-by-expert inside (``fused.gmm_gather``)
           "swiglu"  the gated pair of products (``fused.gmm_swiglu``)
           "layer"   an inference expert layer: gated pair, down projection and
                     weighted top-k combine (``backend.gmm_swiglu``, ``backend.gmm_scatter``)
  pass     "forward" (inference) or "train" (forward, input and weight gradients)
  z        experts; rows are routed to them by ``routing``
  tokens, top_k   rows = tokens * top_k
  k, n     contraction and output columns of the first product (multiples of 8)
  trans_b  weights stored [z, n, k] instead of [z, k, n]
  sizes    "device" or "host": where batch_sizes lives
  routing  "even" (uniform popularity), "skewed" (Dirichlet(1) popularity) or "zipf"
           (Zipf(1.1) popularity with a fifth of the experts idle)

Activations and gradients are ~N(0, 1), weights ~N(0, 0.02), all bf16.
"""
import math

import numpy as np
import torch

from grouped_gemm import ops
from grouped_gemm_b200 import backend, fused

WEIGHT_STD = 0.02


def _case(name, op, pass_, z, tokens, top_k, k, n, trans_b, sizes, routing):
    case = {"op": op, "pass": pass_, "z": z, "tokens": tokens, "top_k": top_k, "k": k, "n": n, "trans_b": trans_b,
            "sizes": sizes, "routing": routing}
    if name is not None:
        case["name"] = name
    return case


def listed():
    return [
        # The smallest training call of the tests: launches and host work are all of it.
        # batch_sizes on the host, where the default build of the original wants them.
        _case("tiny_train", "gmm", "train", 4, 512, 1, 128, 128, False, "host", "even"),
        # The top of the original's own test grid, transposed weights.
        _case("small_train_transposed", "gmm", "train", 16, 2048, 1, 256, 512, True, "device", "skewed"),
        # Sizes that fit no tile: ragged experts, column counts that are multiples of 8 only.
        _case("odd_train", "gmm", "train", 7, 3001, 1, 1000, 2504, False, "device", "skewed"),
        # Token generation, 8 large experts: 32 sequences, two experts each.
        _case("decode_large_experts", "gmm", "forward", 8, 32, 2, 4096, 14336, False, "device", "skewed"),
        # Token generation, 256 small experts: 128 sequences, eight experts each.
        _case("decode_many_experts", "gmm", "forward", 256, 128, 8, 7168, 2048, True, "device", "zipf"),
        # One decode step of a whole expert layer.
        _case("layer_decode", "layer", "forward", 8, 64, 2, 4096, 14336, False, "device", "skewed"),
        # A prompt of 4096 tokens through a whole expert layer.
        _case("layer_prefill", "layer", "forward", 8, 4096, 2, 4096, 14336, False, "device", "skewed"),
        # Training of a gathered projection: the permuted activations never exist.
        _case("gather_train", "gather", "train", 8, 8192, 2, 4096, 14336, False, "device", "skewed"),
        # Training of a gated projection.
        _case("swiglu_train", "swiglu", "train", 8, 8192, 2, 4096, 14336, False, "device", "skewed"),
        # The benchmark's up-projection: forward, input gradient, weight gradient.
        _case("large_experts_train", "gmm", "train", 8, 16384, 2, 4096, 14336, False, "device", "skewed"),
        # Many small experts, a fifth of them empty.
        _case("many_experts_train", "gmm", "train", 256, 8192, 8, 7168, 2048, False, "device", "zipf"),
        # The expert-parallel benchmark's whole job on one GPU.
        _case("largest_train", "gmm", "train", 64, 65536, 4, 6144, 10752, False, "device", "even"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


_MAX_FLOPS = 1.0e14      # of the largest listed case
_MAX_ELEMENTS = 1.5e10   # bf16 values of a case's tensors and results


def draw(rng):
    """A case of the same ranges: every operation and pass, 1 .. 256 experts, 16 rows to
    a quarter of a million, rows and columns of any multiple of 8 up to 14336."""
    while True:
        op, pass_ = rng.choice([("gmm", "train"), ("gmm", "train"), ("gmm", "forward"), ("gather", "train"),
                                ("swiglu", "train"), ("layer", "forward")])
        z = _log_int(rng, 1, 256)
        top_k = min(z, rng.choice([1, 2, 4, 8]))
        tokens = _log_int(rng, 16, 65536)
        k = 8 * _log_int(rng, 8, 1792)
        n = 8 * _log_int(rng, 8, 1792)
        routing = rng.choice(["even", "skewed", "zipf"])
        if routing == "zipf" and z - z // 5 < top_k:
            continue
        case = _case(None, op, pass_, z, tokens, top_k, k, n, rng.random() < 0.5, rng.choice(["device", "device", "host"]),
                     routing)
        rows = tokens * top_k
        weights = z * k * n * {"gmm": 1, "gather": 1, "swiglu": 2, "layer": 3}[op]
        elements = weights * (2 if pass_ == "train" else 1) + rows * 2 * (k + n)
        if rows <= 262144 and elements <= _MAX_ELEMENTS and work(case)["flops"] <= _MAX_FLOPS:
            return case


def _popularity(case, seed):
    """Share of the rows that each expert is expected to get."""
    z = case["z"]
    rng = np.random.RandomState(seed & 0x7FFFFFFF)
    if case["routing"] == "even":
        p = np.full(z, 1.0 / z)
    elif case["routing"] == "skewed":
        p = rng.dirichlet(np.ones(z)) + 1e-4 / z
    else:
        p = np.arange(1, z + 1, dtype=np.float64) ** -1.1
        p[z - z // 5:] = 0.0
        p = rng.permutation(p)
    return p / p.sum()


def _route(case, seed, device):
    """(batch_sizes int64 [z], source token of every row sorted by expert)."""
    gen = torch.Generator(device=device).manual_seed(seed + 1)
    p = torch.from_numpy(_popularity(case, seed)).float().to(device)
    top_k = case["top_k"]
    if top_k == 1:
        experts = torch.multinomial(p, case["tokens"], replacement=True, generator=gen)
    else:
        # top_k different experts per token, drawn by popularity
        noise = torch.rand(case["tokens"], case["z"], generator=gen, device=device).clamp_min_(1e-20)
        scores = torch.where(p > 0, p.log() - (-noise.log()).log(), -math.inf)
        experts = scores.topk(top_k, dim=1).indices.reshape(-1)
    order = torch.argsort(experts, stable=True)
    sizes = torch.bincount(experts, minlength=case["z"])
    return sizes, torch.div(order, top_k, rounding_mode="floor")


def prepare(case, seed):
    device = "cuda"
    z, k, n, tokens = case["z"], case["k"], case["n"], case["tokens"]
    rows = tokens * case["top_k"]
    gen = torch.Generator(device=device).manual_seed(seed)
    sizes, source = _route(case, seed, device)

    def normal(*shape, std=1.0):
        out = torch.empty(*shape, dtype=torch.bfloat16, device=device)
        return out.normal_(0.0, std, generator=gen)

    def weights(rows_, cols):
        shape = (z, cols, rows_) if case["trans_b"] else (z, rows_, cols)
        return normal(*shape, std=WEIGHT_STD)

    state = {"op": case["op"], "train": case["pass"] == "train", "trans_b": case["trans_b"],
             "sizes": sizes.cpu() if case["sizes"] == "host" else sizes, "b": weights(k, n)}
    if case["op"] in ("swiglu", "layer"):
        state["b2"] = weights(k, n)
    if case["op"] == "layer":
        state["down"] = weights(n, k)
        state["row_weight"] = torch.rand(rows, generator=gen, device=device)
    if case["op"] in ("gather", "layer"):
        state["source"] = source
        state["x"] = normal(tokens, k)
    else:
        state["x"] = normal(rows, k)
    if state["train"]:
        state["grad"] = normal(rows, n)
        for name in ("x", "b", "b2"):
            if name in state:
                state[name].requires_grad_(True)
    return state


def run(state):
    op, x, b, sizes, trans_b = state["op"], state["x"], state["b"], state["sizes"], state["trans_b"]
    if op == "layer":
        hidden = backend.gmm_swiglu(x.index_select(0, state["source"]), b, state["b2"], sizes, trans_b=trans_b)
        out = torch.zeros_like(x)
        backend.gmm_scatter(hidden, state["down"], sizes, out, state["source"], trans_b=trans_b,
                            row_weight=state["row_weight"], accumulate=True)
        return out
    leaves = (x, b)
    if op == "gmm":
        out = ops.gmm(x, b, sizes, trans_b)
    elif op == "gather":
        out = fused.gmm_gather(x, state["source"], b, sizes, trans_b)
    else:
        out = fused.gmm_swiglu(x, b, state["b2"], sizes, trans_b)
        leaves = (x, b, state["b2"])
    if not state["train"]:
        return out
    return (out.detach(),) + torch.autograd.grad(out, leaves, state["grad"])


def work(case):
    """Every input once and every output once; the products that the results are made of
    (a gated product computed a second time in the backward pass does not count).
    Weights of experts that got no row need not be read."""
    z, k, n, tokens, top_k = case["z"], case["k"], case["n"], case["tokens"], case["top_k"]
    rows = tokens * top_k
    active = float(np.sum(1.0 - (1.0 - _popularity(case, 0)) ** rows))
    product = 2.0 * rows * k * n
    one, used = k * n * z, k * n * active
    if case["op"] == "layer":
        return {"bytes": 2.0 * (2 * tokens * k + 3 * used) + 12.0 * rows + 8.0 * z, "flops": 3 * product}
    inputs = tokens if case["op"] == "gather" else rows
    pairs = 2 if case["op"] == "swiglu" else 1
    total = inputs * k + pairs * used + rows * n
    if case["pass"] == "train":
        total += rows * n + inputs * k + pairs * one
    indices = 8.0 * rows if case["op"] == "gather" else 0.0
    return {"bytes": 2.0 * total + indices + 8.0 * z,
            "flops": pairs * product * (3 if case["pass"] == "train" else 1)}


def _product64(x, w, sizes):
    """Rows of ``x`` grouped by ``sizes`` times ``w[i]`` each, in 64 bits; idle experts are skipped."""
    out = torch.empty(x.shape[0], w.shape[2], dtype=torch.float64, device=x.device)
    start = 0
    for i, size in enumerate(sizes):
        if size:
            torch.mm(x[start:start + size].double(), w[i].double(), out=out[start:start + size])
        start += size
    return out


def _weight_grad64(x, grad, sizes, transposed):
    shape = (len(sizes), grad.shape[1], x.shape[1]) if transposed else (len(sizes), x.shape[1], grad.shape[1])
    out = torch.zeros(shape, dtype=torch.float64, device=x.device)
    start = 0
    for i, size in enumerate(sizes):
        if size:
            rows, cols = (grad, x) if transposed else (x, grad)
            torch.mm(rows[start:start + size].double().t(), cols[start:start + size].double(), out=out[i])
        start += size
    return out


def exact(case, seed):
    """What ``run`` returns, computed in 64 bits from the same bf16 inputs."""
    state = prepare(case, seed)
    state = {key: v.detach() if isinstance(v, torch.Tensor) else v for key, v in state.items()}
    op, x, trans_b = state["op"], state["x"], state["trans_b"]
    sizes = [int(s) for s in state["sizes"].tolist()]
    # weights as [z, in, out]
    b, b2, down = (state[key].transpose(1, 2) if trans_b and key in state else state.get(key) for key in ("b", "b2", "down"))
    rows = x.index_select(0, state["source"]) if op in ("gather", "layer") else x
    out = _product64(rows, b, sizes)
    if op in ("swiglu", "layer"):
        gate, up = out, _product64(rows, b2, sizes)
        out = torch.nn.functional.silu(gate) * up
    if op == "layer":
        y = _product64(out, down, sizes) * state["row_weight"].double()[:, None]
        return torch.zeros(x.shape, dtype=torch.float64, device=x.device).index_add_(0, state["source"], y)
    if case["pass"] != "train":
        return out
    grad = state["grad"]
    if op == "swiglu":
        s = torch.sigmoid(gate)
        d_up = grad * gate * s
        d_gate = grad * up * s * (1.0 + gate * (1.0 - s))
        del s, gate, up
        x_grad = _product64(d_gate, b.transpose(1, 2), sizes) + _product64(d_up, b2.transpose(1, 2), sizes)
        return out, x_grad, _weight_grad64(rows, d_gate, sizes, trans_b), _weight_grad64(rows, d_up, sizes, trans_b)
    x_grad = _product64(grad, b.transpose(1, 2), sizes)
    if op == "gather":
        x_grad = torch.zeros(x.shape, dtype=torch.float64, device=x.device).index_add_(0, state["source"], x_grad)
    return out, x_grad, _weight_grad64(rows, grad, sizes, trans_b)


def tolerance(case):
    """Four times the distance from the same path in 64 bits.  A single product is one
    rounding to bf16 of an fp32 sum (1.66e-3; largest element 3.9e-3).  The other paths
    round more than once: rows of top_k experts added in bf16 in memory (top_k 8: 4.3e-3,
    largest 2.7e-2), or a gradient that went through a bf16 intermediate (3.0e-3, 1.6e-2)."""
    if case["op"] == "gmm":
        return {"rel": 7e-3, "max": 1.6e-2}
    return {"rel": 1.7e-2, "max": 1.1e-1}
