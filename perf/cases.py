"""The work that performance is measured on: one case per path that a user of the pairwise operators runs in earnest.

``listed()`` holds the cases, ``draw(rng)`` gives another of the same ranges, ``prepare`` makes what a program has in
hand before the call, ``run`` is one pass through the public operators, ``work`` the bytes and operations that the pass
cannot do without, ``tolerance`` the error that another correct evaluation at the same precision shows and ``exact`` the
outputs in 64 bits.
"""
import math

import torch

import torchpairwise_b200 as tp

tp.load_torch_ops()
OPS = torch.ops.torchpairwise

F32, F64, BF16 = torch.float32, torch.float64, torch.bfloat16


def listed():
    return [
        # few-shot classification head: the queries of one episode against the class prototypes, both trained through
        # the distance; four small launches and the host path around them are the whole cost
        dict(name="prototypes", kind="prototypes", n1=75, n2=5, d=64),
        # the ordinary small matrix, L1, forward and backward
        dict(name="manhattan", kind="manhattan", n1=1024, n2=2048, d=128),
        # batched point-to-point L_p loss at full size, p = 3: the headline workload, through the dispatcher's operator
        dict(name="minkowski3", kind="minkowski3", b=16, n1=4096, n2=4096, d=256),
        # batched Chebyshev, forward and backward
        dict(name="chebyshev", kind="chebyshev", b=16, n1=4096, n2=4096, d=256),
        # standardised Euclidean in double precision on ragged statistics tables, forward and backward
        dict(name="seuclidean_f64", kind="seuclidean_f64", n1=1500, n2=1301, d=75),
        # similarity search over long binary descriptors, through the dispatcher's operator
        dict(name="jaccard", kind="boolean", metric="jaccard", n1=65536, n2=16384, d=1024),
        # the same over short fingerprints whose rows fill no whole word
        dict(name="hamming_ragged", kind="boolean", metric="hamming", n1=30011, n2=10007, d=167),
        # large dense distance matrix, forward only (clustering, retrieval)
        dict(name="sqeuclidean_dense", kind="sqeuclidean_dense", n1=131072, n2=16384, d=512),
        # Euclidean loss between batched feature sets, forward and backward
        dict(name="euclidean_train", kind="euclidean_train", b=16, n1=4096, n2=4096, d=256),
        # cosine loss between the embeddings of two ragged batches in bfloat16, forward and backward
        dict(name="cosine_bf16", kind="cosine_bf16", n1=5000, n2=4111, d=768),
        # directed Hausdorff between point clouds and their perturbed copies, forward and backward
        dict(name="hausdorff", kind="hausdorff", b=64, n1=8192, n2=8192, d=3),
        # k nearest neighbours of a query set in a reference set
        dict(name="neighbours", kind="neighbours", n1=50000, n2=20000, d=128, k=10),
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, evenly spread over its logarithm."""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["prototypes", "manhattan", "minkowski3", "chebyshev", "seuclidean_f64", "boolean", "sqeuclidean_dense",
                       "euclidean_train", "cosine_bf16", "hausdorff", "neighbours"])
    c = dict(kind=kind)
    if kind == "prototypes":
        c.update(n1=_log(rng, 25, 600), n2=rng.randint(5, 60), d=rng.choice([64, 100, 128, 192]))
    elif kind == "manhattan":
        c.update(n1=_log(rng, 256, 2048), n2=_log(rng, 256, 2048), d=_log(rng, 32, 128))
    elif kind in ("minkowski3", "chebyshev", "euclidean_train"):
        # from a few ragged sets to the full batch; features mostly a multiple of four, as layer widths are
        d = rng.choice([64, 100, 128, 192, 256, rng.randint(60, 255)])
        c.update(b=rng.randint(1, 16), n1=_log(rng, 300, 4096), n2=_log(rng, 300, 4096), d=d)
    elif kind == "seuclidean_f64":
        c.update(n1=_log(rng, 200, 1500), n2=_log(rng, 200, 1300), d=_log(rng, 10, 75))
    elif kind == "boolean":
        c.update(metric=rng.choice(["hamming", "jaccard"]), n1=_log(rng, 2000, 65536), n2=_log(rng, 2000, 16384),
                 d=rng.choice([166, 512, 1024, rng.randint(150, 1024)]))
    elif kind == "sqeuclidean_dense":
        c.update(n1=_log(rng, 4000, 131072), n2=_log(rng, 1000, 16384), d=rng.choice([96, 128, 256, 384, 512, rng.randint(64, 511)]))
    elif kind == "cosine_bf16":
        c.update(n1=_log(rng, 512, 5000), n2=_log(rng, 512, 4100), d=rng.choice([256, 384, 512, 768]))
    elif kind == "hausdorff":
        c.update(b=rng.randint(4, 64), n1=_log(rng, 500, 8192), n2=_log(rng, 500, 8192), d=rng.choice([2, 3, 3]))
    else:
        c.update(n1=_log(rng, 2000, 50000), n2=_log(rng, 2000, 20000), d=rng.choice([64, 96, 128]), k=rng.randint(1, 16))
    return c


def _randn(g, *shape, dtype=F32):
    return torch.randn(*shape, generator=g, device="cuda", dtype=dtype)


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    kind, n1, n2, d = case["kind"], case["n1"], case["n2"], case["d"]
    if kind == "boolean":
        return dict(kind=kind, metric=case["metric"], x1=torch.rand(n1, d, generator=g, device="cuda") < 0.1,
                    x2=torch.rand(n2, d, generator=g, device="cuda") < 0.1)
    if kind in ("sqeuclidean_dense", "neighbours"):
        return dict(kind=kind, x1=_randn(g, n1, d), x2=_randn(g, n2, d), k=case.get("k"))
    if kind == "hausdorff":
        # points of the unit cube [-1, 1]^d and perturbed points of the same cloud (drawn again where x2 has more)
        b, m = case["b"], max(n1, n2)
        cloud = torch.rand(b, m, d, generator=g, device="cuda") * 2 - 1
        x1 = cloud[:, :n1].contiguous().unsqueeze(1).requires_grad_()
        x2 = (cloud[:, :n2] + 0.05 * _randn(g, b, n2, d)).unsqueeze(1).requires_grad_()
        return dict(kind=kind, x1=x1, x2=x2, grad=_randn(g, b, 1, 1))
    lead = (case["b"],) if "b" in case else ()
    dtype = {"seuclidean_f64": F64, "cosine_bf16": BF16}.get(kind, F32)
    s = dict(kind=kind, x1=_randn(g, *lead, n1, d, dtype=dtype).requires_grad_(), x2=_randn(g, *lead, n2, d, dtype=dtype).requires_grad_(),
             grad=_randn(g, *lead, n1, n2, dtype=dtype))
    if kind == "seuclidean_f64":
        s["V"] = torch.rand(d, generator=g, device="cuda", dtype=F64) + 0.5
    return s


def run(state):
    kind, x1, x2 = state["kind"], state["x1"], state["x2"]
    if kind == "boolean":
        return OPS.jaccard_distances(x1, x2) if state["metric"] == "jaccard" else OPS.hamming_distances(x1, x2)
    if kind == "sqeuclidean_dense":
        return tp.sqeuclidean_distances(x1, x2)
    if kind == "neighbours":
        return tp.pairwise_argkmin(x1, x2, state["k"], "euclidean")
    if kind == "prototypes":
        out = tp.euclidean_distances(x1, x2)
    elif kind == "manhattan":
        out = tp.manhattan_distances(x1, x2)
    elif kind == "minkowski3":
        out = OPS.minkowski_distances(x1, x2, 3.0)
    elif kind == "chebyshev":
        out = tp.chebyshev_distances(x1, x2)
    elif kind == "seuclidean_f64":
        out = tp.seuclidean_distances(x1, x2, state["V"])
    elif kind == "euclidean_train":
        out = tp.euclidean_distances(x1, x2)
    elif kind == "cosine_bf16":
        out = tp.cosine_distances(x1, x2)
    else:
        out, at1, at2 = tp.directed_hausdorff_distances(x1, x2)
        g1, g2 = torch.autograd.grad(out, (x1, x2), state["grad"])
        return out.detach(), at1, at2, g1, g2
    g1, g2 = torch.autograd.grad(out, (x1, x2), state["grad"])
    return out.detach(), g1, g2


def work(case):
    kind, b, n1, n2, d = case["kind"], case.get("b", 1), case["n1"], case["n2"], case["d"]
    pairs, inputs = b * n1 * n2, b * (n1 + n2) * d
    if kind == "boolean":
        return dict(bytes=inputs + 4 * pairs, flops=2 * pairs * d)
    if kind == "sqeuclidean_dense":
        return dict(bytes=4 * inputs + 4 * pairs, flops=2 * pairs * d)
    if kind == "neighbours":
        return dict(bytes=4 * inputs + 12 * n1 * case["k"], flops=2 * pairs * d)
    if kind == "hausdorff":
        # the direct evaluation: subtract and multiply-add per coordinate and a minimum per pair of points
        return dict(bytes=8 * inputs + 28 * b, flops=pairs * (3 * d + 1))
    # forward and backward: the output written and, with the upstream gradient, read; inputs read and gradients written
    size = {"seuclidean_f64": 8, "cosine_bf16": 2}.get(kind, 4)
    per = {"manhattan": 5, "minkowski3": 10, "chebyshev": 2, "seuclidean_f64": 8}.get(kind, 6)
    return dict(bytes=size * (2 * inputs + 2 * pairs), flops=per * pairs * d)


# Largest relative error (2-norm) of outputs and gradients against a float64 evaluation of the same inputs, times four.
# Chebyshev: the float32 differences tie where the float64 ones do not, so the figure is that of inputs without ties.
_REL = {"prototypes": 1e-6, "manhattan": 4e-6, "minkowski3": 5e-6, "chebyshev": 3e-6, "seuclidean_f64": 6e-15, "sqeuclidean_dense": 1e-6,
        "euclidean_train": 2e-6, "cosine_bf16": 7e-3, "hausdorff": 1e-6, "neighbours": 1.5e-6}


def tolerance(case):
    kind = case["kind"]
    if kind == "boolean":
        return "exact"
    # neighbours: 1e-4 of the indices trade places with a neighbour whose distance agrees to float32 rounding
    return {"rel": _REL[kind], "differ": 5e-4} if kind == "neighbours" else {"rel": _REL[kind]}


def _differences(x1, x2, grad, p, w):
    """A batch's distances by direct differences, (sum w |x - y|^p)^(1/p), and their gradients; x1 a block of rows at a time."""
    out, g1, g2 = x1.new_empty(x1.size(0), x2.size(0)), torch.empty_like(x1), torch.zeros_like(x2)
    rows = max(1, (1 << 26) // (x2.size(0) * x2.size(1)))
    for i in range(0, x1.size(0), rows):
        at = slice(i, i + rows)
        d = x1[at, None] - x2
        if p == math.inf:
            # a coordinate attains the maximum where its float32 difference does: that is what the inputs' type resolves
            d = d.float().double()
            out[at] = d.abs().amax(2)
            t = torch.where(d.abs() == out[at, :, None], d.sign(), 0.0)
            c = grad[at]
        else:
            t = d.sign() if p == 1 else d * d.abs() ** (p - 2) if p > 2 else d
            t = t if w is None else t * w
            out[at] = (t * d).sum(2) ** (1 / p)
            c = grad[at] if p == 1 else grad[at] / out[at] ** (p - 1)
        t = t * c[..., None]
        g1[at] = t.sum(1)
        g2 -= t.sum(0)
    return out, g1, g2


def exact(case, seed):
    s = prepare(case, seed)
    kind = case["kind"]
    if kind == "boolean":
        return None
    x1, x2 = s["x1"].detach().double(), s["x2"].detach().double()
    if kind == "sqeuclidean_dense":
        out = torch.addmm(x1.square().sum(1)[:, None], x1, x2.T, alpha=-2)
        return out.add_(x2.square().sum(1)).clamp_(min=0)
    if kind == "neighbours":
        best = []
        for a in x1.split(8192):
            d = torch.addmm(a.square().sum(1)[:, None], a, x2.T, alpha=-2).add_(x2.square().sum(1)).clamp_(min=0).sqrt_()
            best.append(d.topk(case["k"], largest=False).values)
        return None, torch.cat(best)
    grad = s["grad"].double()
    if kind == "hausdorff":
        out, g1, g2 = torch.empty_like(grad), torch.zeros_like(x1), torch.zeros_like(x2)
        for b in range(x1.size(0)):
            nearest, at = sum((x1[b, 0, :, None, c] - x2[b, 0, None, :, c]).square() for c in range(x1.size(3))).min(1)
            m = nearest.argmax()
            out[b] = nearest[m].sqrt()
            g = grad[b, 0, 0] * (x1[b, 0, m] - x2[b, 0, at[m]]) / out[b, 0, 0]
            g1[b, 0, m], g2[b, 0, at[m]] = g, -g
        return out, None, None, g1, g2
    if kind == "cosine_bf16":
        x1.requires_grad_(), x2.requires_grad_()
        out = 1 - (x1 / x1.norm(dim=1, keepdim=True)) @ (x2 / x2.norm(dim=1, keepdim=True)).T
        return out.detach(), *torch.autograd.grad(out, (x1, x2), grad)
    p = {"manhattan": 1, "minkowski3": 3, "chebyshev": math.inf}.get(kind, 2)
    w = 1 / s["V"] if kind == "seuclidean_f64" else None
    if "b" not in case:
        return _differences(x1, x2, grad, p, w)
    return [torch.stack(v) for v in zip(*(_differences(x1[b], x2[b], grad[b], p, w) for b in range(case["b"])))]
