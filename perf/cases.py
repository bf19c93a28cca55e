"""Performance cases of the framework: what a program that trains, evaluates and samples probabilistic circuits has
it do, through the public entry points of `lvd_pg_b200.api`.

Every case is one call (or the pair of calls that belong together) of one `kind`:

  em        one mini-batch EM step on hard evidence: forward, backward, statistics, update
  em_soft   the same on per-category log-weights (soft evidence)
  ll        log-likelihoods of a data set, in batches, with missing values
  kld_adam  KLD + gradient + Adam + re-normalisation of one parameter set (the variational loop)
  kld       KLD and both gradients for a batch of parameter sets (the loss of a PC-VAE)
  sample    hard Gumbel-max samples
  soft      relaxed (Gumbel-softmax) samples, one parameter set per sample
  nflows    per-row normalised flows of every parameter
  mi        pairwise mutual information of a data matrix (the input of Chow-Liu learning)

Circuits are HCLTs with `k` latent states.  "image" trees connect the (y, x, channel) variables of square colour
images the way a Chow-Liu tree of natural images does (mostly to a neighbouring pixel of the same channel, deep);
"random" trees are the shallow random spanning trees of the variational benchmark.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from lvd_pg_b200 import api, structures as st

DEVICE = 0


def listed():
    return [
        # The smallest step anybody takes: 64 binary variables, 16 latent states (a tree-structured Bernoulli model
        # on tabular data).  A chain of small launches; latency counts.
        dict(name="em_tabular", kind="em", tree="random", vars=64, cats=2, k=16, batch=256, missing=0.0),
        # One patch circuit of a 64x64 image model: 8x8x3 pixels, 128 latent states, a batch of 256 images.
        dict(name="em_patch", kind="em", tree="image", vars=192, cats=256, k=128, batch=256, missing=0.0),
        # 32x32x3 images with few latent states: wide and deep, little arithmetic per node.
        dict(name="em_image_narrow", kind="em", tree="image", vars=3072, cats=256, k=32, batch=512, missing=0.0),
        # Wide latent states and a large batch, the shape of the headline training run on 16x16x3 images.
        dict(name="em_image_wide", kind="em", tree="image", vars=768, cats=256, k=256, batch=2048, missing=0.0),
        # Training on the soft outputs of a teacher network: odd sizes everywhere.
        dict(name="em_soft_ragged", kind="em_soft", tree="random", vars=100, cats=33, k=72, batch=300, missing=0.0),
        # Test-set likelihoods with missing values, in batches that do not divide the rows.
        dict(name="ll_missing", kind="ll", tree="random", vars=784, cats=2, k=64, batch=512, rows=5000, missing=0.1),
        # One step of the variational loop on one parameter set.
        dict(name="kld_adam", kind="kld_adam", tree="random", vars=784, cats=2, k=64, batch=1, missing=0.0),
        # Loss and gradients of a PC-VAE batch: one parameter set per example.
        dict(name="kld_batch", kind="kld", tree="random", vars=784, cats=2, k=64, batch=24, missing=0.0),
        # Samples of the model, noise supplied by the caller.
        dict(name="sample_hard", kind="sample", tree="random", vars=784, cats=2, k=64, batch=4096, missing=0.0),
        # Relaxed samples a PC-VAE differentiates through: one parameter set per sample.
        dict(name="sample_soft", kind="soft", tree="random", vars=784, cats=2, k=64, batch=24, missing=0.0),
        # The encoder side of the variational loop: normalised flows of a batch of rows.
        dict(name="norm_flows", kind="nflows", tree="random", vars=784, cats=2, k=64, batch=512, missing=0.0),
        # Structure learning: pairwise mutual information of 32x32x3 images at 32 levels.
        dict(name="pairwise_mi", kind="mi", tree="image", vars=3072, cats=32, k=0, batch=4096, missing=0.0),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["em", "em", "em", "em", "em_soft", "ll", "kld_adam", "kld", "sample", "soft", "nflows", "mi"])
    if kind == "mi":
        cats = rng.choice([2, 4, 8, 16, 32, 64, 128, 256])   # the entry point takes powers of two
        return dict(kind=kind, tree="image", vars=size(64, min(3072, 98304 // cats)), cats=cats, k=0,
                    batch=size(512, 4096), missing=0.0)
    if kind in ("em", "ll"):
        tree = rng.choice(["image", "random"])
        k = size(16, 256)
        v = size(48, min(3072, 768 * 65536 // (k * k)))
        b = size(64, min(2048, 768 * 256 * 2048 // (v * k)))
        case = dict(kind=kind, tree=tree, vars=v, cats=rng.choice([2, 10, 100, 256]), k=k, batch=b,
                    missing=rng.choice([0.0, 0.0, 0.1]))
        if kind == "ll":
            case["rows"] = int(b * rng.uniform(1.0, 4.0))
        return case
    if kind == "em_soft":
        return dict(kind=kind, tree="random", vars=size(24, 400), cats=size(4, 64), k=size(16, 128),
                    batch=size(64, 512), missing=0.0)
    top = {"kld_adam": 1, "kld": 32, "sample": 4096, "soft": 32, "nflows": 512}[kind]
    return dict(kind=kind, tree="random", vars=size(48, 784), cats=rng.choice([2, 5]), k=size(16, 64),
                batch=size(max(1, top // 16), top) if top > 1 else 1, missing=0.0)


# ---- structures: the same for every seed --------------------------------------------------------------
@functools.lru_cache(maxsize=8)
def _tree(tree: str, v: int) -> np.ndarray:
    rng = np.random.default_rng(4)
    if tree == "random":
        return st.root_tree_at_center(v, st.random_spanning_tree(v, rng))
    # neighbouring pixels share more information than the channels of one pixel (weights stand in for the estimate)
    side = math.ceil(math.sqrt(v / 3))
    w = np.full((v, v), 0.0)
    i = np.arange(v)
    x, c = (i // 3) % side, i % 3
    for step, ok, lo, hi in ((3, x + 1 < side, 0.8, 1.0), (3 * side, np.ones(v, bool), 0.8, 1.0), (1, c < 2, 0.6, 0.85)):
        a = i[ok & (i + step < v)]
        w[a, a + step] = w[a + step, a] = rng.uniform(lo, hi, a.size)
    return st.root_tree_at_center(v, st.max_spanning_tree(w))


@functools.lru_cache(maxsize=2)
def _circuit(tree: str, v: int, cats: int, k: int):
    return st.hclt_flat(_tree(tree, v), cats, k, seed=None)


def _sum_edges(case) -> int:
    parent = _tree(case["tree"], case["vars"])
    inner = len(set(int(p) for p in parent if p >= 0))
    return (inner - 1) * case["k"] ** 2 + case["k"]


def _num_params(case) -> int:
    return _sum_edges(case) + case["vars"] * case["k"] * case["cats"]


# ---- inputs ---------------------------------------------------------------------------------------------
def _log_dirichlet(gen, rows: int, cols: int, device) -> torch.Tensor:
    """Log of `rows` Dirichlet(1, ..., 1) draws of dimension `cols`."""
    e = torch.empty(rows, cols, device=device).exponential_(generator=gen).clamp_(min=1e-30)
    return e.div_(e.sum(1, keepdim=True)).log_()


def _params(case, gen, device) -> torch.Tensor:
    """One flat parameter vector: sum groups (k edges each), then leaves."""
    k, cats = case["k"], case["cats"]
    edges = _sum_edges(case)
    return torch.cat([_log_dirichlet(gen, edges // k, k, device).view(-1),
                      _log_dirichlet(gen, case["vars"] * k, cats, device).view(-1)])


def _data(case, rows: int, gen, device) -> torch.Tensor:
    """uint8 [vars, rows]: smooth colour images quantised to `cats` levels, or binary columns."""
    v, cats = case["vars"], case["cats"]
    if case["tree"] == "random":
        p = torch.rand(v, 1, generator=gen, device=device) * 0.8 + 0.1
        u = torch.rand(v, rows, generator=gen, device=device)
        if cats == 2:
            return (u < p).to(torch.uint8)
        return (u ** (2 * p) * cats).to(torch.int64).clamp_(max=cats - 1).to(torch.uint8)
    side = math.ceil(math.sqrt(v / 3))
    out = torch.empty(v, rows, dtype=torch.uint8, device=device)
    for r0 in range(0, rows, 1024):
        n = min(1024, rows - r0)
        z = torch.randn(4, side, side, n, generator=gen, device=device)
        for _ in range(8):   # eight binomial passes: about two pixels of blur
            for d in (1, 2):
                z = 0.5 * z + 0.25 * (z.roll(1, d) + z.roll(-1, d))
        z = z * 7.0           # back to unit scale
        img = 0.9 * z[:1] + 0.45 * z[1:]                       # [channel, y, x, n], channels correlated 0.8
        lev = ((img * 50.0 + 128.0).clamp_(0, 255) * (cats / 256.0)).to(torch.uint8).clamp_(max=cats - 1)
        out[:, r0:r0 + n] = lev.permute(1, 2, 0, 3).reshape(-1, n)[:v]
    return out


def prepare(case, seed):
    dev = torch.device("cuda", DEVICE)
    gen = torch.Generator(device=dev).manual_seed(seed)
    kind, B = case["kind"], case["batch"]
    s = {"case": case}
    if kind == "mi":
        s["data"] = api.DeviceData.from_colmajor(_data(case, B, gen, dev))
        return s
    m = s["m"] = api.CuMetaBitsProbCircuit(_circuit(case["tree"], case["vars"], case["cats"], case["k"]), DEVICE)
    theta = s["theta"] = _params(case, gen, dev)
    api.update_parameters(m, theta)
    S = B
    if kind in ("em", "em_soft"):
        rows = 4 * B
        if kind == "em":
            miss = None
            if case["missing"]:
                miss = (torch.rand(case["vars"], rows, generator=gen, device=dev) < case["missing"]).to(torch.uint8)
            s["data"] = api.DeviceData.from_colmajor(_data(case, rows, gen, dev), miss)
        else:
            s["soft"] = _log_dirichlet(gen, rows * case["vars"], case["cats"], dev).view(
                rows, case["vars"], case["cats"]).permute(2, 1, 0).contiguous().permute(2, 1, 0)
        s["ids"] = (torch.randperm(rows, generator=gen, device=dev) + 1).to(torch.int32)
        s["next"], s["ll"] = 0, torch.zeros(1, device=dev)
        m.workspace(B)
    elif kind == "ll":
        rows = case["rows"]
        miss = None
        if case["missing"]:
            miss = (torch.rand(case["vars"], rows, generator=gen, device=dev) < case["missing"]).to(torch.uint8)
        s["data"] = api.DeviceData.from_colmajor(_data(case, rows, gen, dev), miss)
        m.workspace(B)
    elif kind == "kld_adam":
        s["q"] = _params(case, gen, dev)
        s["opt"] = api.KldAdam(m, s["q"], theta, lr=1e-2)
    elif kind == "kld":
        s["p1"] = torch.stack([_params(case, gen, dev) for _ in range(S)])
        s["p2"] = torch.stack([_params(case, gen, dev) for _ in range(S)])
        m.workspace(1)
    elif kind == "sample":
        shp = api.noise_shapes(m, S)
        s["u_sum"] = torch.rand(shp[0], generator=gen, device=dev)
        s["u_leaf"] = torch.rand(shp[1], generator=gen, device=dev)
        m.workspace(1)
    elif kind == "soft":
        s["params"] = torch.stack([_params(case, gen, dev) for _ in range(S)])
        s["u"] = torch.rand(S, m.num_inner_params, generator=gen, device=dev)
        m.workspace(1)
    elif kind == "nflows":
        s["data"] = api.DeviceData.from_colmajor(_data(case, B, gen, dev))
        m.workspace(B)
    return s


def run(state):
    case = state["case"]
    kind, B = case["kind"], case["batch"]
    if kind == "mi":
        return api.pairwise_mi(state["data"], case["cats"], 0.1, DEVICE)
    m = state["m"]
    if kind in ("em", "em_soft"):
        b = state["next"]
        state["next"] = (b + 1) % 4
        ids = state["ids"][b * B:(b + 1) * B]
        if kind == "em":
            api.em_step(m, state["data"], ids, 1, B, 0.1, 0.9, 0.0, None, state["ll"])
        else:
            api.em_step_ex(m, None, state["soft"], None, ids, 1, B, 0.1, 0.9, ll_sum=state["ll"])
        return {"ll": state["ll"], "theta": api.vectorize_parameters(m, state["theta"])}
    if kind == "ll":
        return api.loglikelihoods(m, state["data"], B)
    if kind == "kld_adam":
        opt = state["opt"]
        return {"kld": opt.step(), "q": opt.q, "m": opt.m, "v": opt.v}
    if kind == "kld":
        out, reuse = api.kld(m, state["p1"], state["p2"])
        g1, g2 = api.kld_backward(m, reuse=reuse)
        return {"kld": out, "g1": g1, "g2": g2}
    if kind == "sample":
        return api.sample(m, state["theta"], state["u_sum"], state["u_leaf"])
    if kind == "soft":
        return api.gumbel_sample(m, state["params"], case["vars"], case["cats"], 0.7, u=state["u"])
    return api.per_sample_normalized_flows(m, state["data"], None, B)


def work(case):
    """What one pass cannot do without: inputs read once, outputs written once, the contractions of the sum layers."""
    kind, v, c, k, B = case["kind"], case["vars"], case["cats"], case["k"], case["batch"]
    if kind == "mi":
        return {"bytes": B * v + 4.0 * v * v, "flops": float(v * c) ** 2 * B}
    edges, P = float(_sum_edges(case)), float(_num_params(case))
    rows = case.get("rows", B)
    data = rows * v * (2.0 if case["missing"] else 1.0)
    return {
        "em": {"bytes": data + 8.0 * P, "flops": 6.0 * B * edges},
        "em_soft": {"bytes": 4.0 * B * v * c + 8.0 * P, "flops": 6.0 * B * edges},
        "ll": {"bytes": data + 4.0 * P + 4.0 * rows, "flops": 2.0 * rows * edges},
        "kld_adam": {"bytes": 28.0 * P, "flops": 0.0},
        "kld": {"bytes": 16.0 * B * P, "flops": 0.0},
        "sample": {"bytes": 4.0 * B * (edges / k + 1) + 4.0 * B * v * (c + 1) + 4.0 * P, "flops": 0.0},
        "soft": {"bytes": 4.0 * B * (P + edges + v * c), "flops": 0.0},
        "nflows": {"bytes": data + 4.0 * B * P + 4.0 * P, "flops": 0.0},
    }[kind]


# ---- the same outputs in 64 bits, by plain torch ----------------------------------------------------------
class _Tree:
    """The HCLT over one latent tree: children before parents, and where a variable's parameters lie in the flat vector
    (sum blocks by layer and then in post-order, row = latent state of the variable, column = state of its child;
    leaves in post-order behind them)."""

    def __init__(self, case):
        parent, k, c = _tree(case["tree"], case["vars"]), case["k"], case["cats"]
        self.k, self.cats, self.ch = k, c, [[] for _ in parent]
        for y, p in enumerate(parent):
            if p >= 0:
                self.ch[p].append(y)
        self.root = int(np.nonzero(parent < 0)[0][0])
        self.order, stack = [], [self.root]     # parents before children, last child first
        while stack:
            y = stack.pop()
            self.order.append(y)
            stack.extend(self.ch[y])
        self.order.reverse()
        self.inner = [y for y in self.order if self.ch[y]]
        layer, key = {}, []
        for pos, y in enumerate(self.order):
            lay = max((layer[x] for x in self.ch[y]), default=0)
            layer[y] = lay + (2 if len(self.ch[y]) > 1 else 1) if self.ch[y] else 0
            if self.ch[y]:
                key.append((layer[y], pos, y))
        self.sum_at, at = {}, 0
        for _, _, y in sorted(key):
            r = 1 if y == self.root else k
            self.sum_at[y] = (at, r)
            at += r * k
        self.leaf_at = {y: at + i * k * c for i, y in enumerate(self.order)}

    def sums(self, p, y):
        """[..., r, k] of a parameter tensor [..., P]."""
        at, r = self.sum_at[y]
        return p[..., at:at + r * self.k].unflatten(-1, (r, self.k))

    def leaf(self, p, y):
        """[..., k, cats]"""
        at = self.leaf_at[y]
        return p[..., at:at + self.k * self.cats].unflatten(-1, (self.k, self.cats))

    def up(self, theta, leaf_value):
        """Per inner variable: exp(x - max) [B, k] of its children's log-values, sums [B, r]; and the root's log-values."""
        out, kept = {}, {}
        for y in self.order:
            if not self.ch[y]:
                out[y] = leaf_value(y)
                continue
            x = leaf_value(y) + sum(out.pop(c) for c in self.ch[y])
            top = x.max(1, keepdim=True).values
            e = (x - top).exp_()
            s = e @ self.sums(theta, y).exp().t()
            kept[y] = (e, s)
            out[y] = s.log() + top
        return kept, out[self.root][:, 0]

    def down(self, theta, kept):
        """Yields (variable, flow of its leaf nodes [B, k], flow of its sum nodes over their sums [B, r] or None)."""
        flow = {self.root: torch.ones_like(kept[self.root][1])}
        for y in reversed(self.order):
            f = flow.pop(y)
            if not self.ch[y]:
                yield y, f, None
                continue
            e, s = kept[y]
            g = f / s
            f = e * (g @ self.sums(theta, y).exp())
            for c in self.ch[y]:
                flow[c] = f
            yield y, f, g


def _exact_em(case, s, t, theta):
    B, c = case["batch"], case["cats"]
    ids = (s["ids"][:B] - 1).long()
    if case["kind"] == "em_soft":
        soft = s["soft"][ids].double()

        def value(y):
            return torch.logsumexp(soft[:, y, None, :] + t.leaf(theta, y)[None], 2)
    else:
        x = s["data"].t[:, ids].long()
        miss = None if s["data"].miss is None else s["data"].miss[:, ids].bool()

        def value(y):
            v = t.leaf(theta, y)[:, x[y]].t()
            return v if miss is None else v.masked_fill(miss[y][:, None], 0.0)
    kept, ll = t.up(theta, value)
    new = torch.empty_like(theta)

    def blend(old, share):
        return (0.9 * old.exp() + 0.1 * share).log()

    for y, f, g in t.down(theta, kept):
        if g is not None:
            w = t.sums(theta, y)
            stat = w.exp() * (g.t() @ kept.pop(y)[0]) + 0.1 / t.k
            t.sums(new, y).copy_(blend(w, stat / stat.sum(1, keepdim=True)))
        w = t.leaf(theta, y)
        if case["kind"] == "em_soft":
            e = soft[:, y, None, :] + w[None]
            stat, lost = ((e - torch.logsumexp(e, 2, keepdim=True)).exp() * f[:, :, None]).sum(0), 0.0
        else:
            keep = 1.0 if miss is None else (~miss[y]).double()[:, None]
            stat = torch.zeros(c, t.k, dtype=torch.float64, device=theta.device).index_add_(0, x[y], f * keep).t()
            lost = (f * (1.0 - keep)).sum(0)[:, None]
        total = stat.sum(1, keepdim=True) + lost + 0.1
        t.leaf(new, y).copy_(blend(w, (stat + 0.1 / c + lost * w.exp()) / total))
    return {"ll": ll.sum()[None], "theta": new}


def _exact_kld(t, p1, p2):
    """KLD(p1 || p2) per set, and the gradients with respect to both ([S, P])."""
    up, below = {}, {}
    for y in t.order:
        a, b = t.leaf(p1, y), t.leaf(p2, y)
        v = (a.exp() * (a - b)).sum(-1)
        if t.ch[y]:
            below[y] = v = v + sum(up.pop(c) for c in t.ch[y])
            a, b = t.sums(p1, y), t.sums(p2, y)
            v = (a.exp() * (v[:, None, :] + a - b)).sum(-1)
        up[y] = v
    g1, g2 = torch.empty_like(p1), torch.empty_like(p2)
    grad = {t.root: torch.ones_like(up[t.root])}
    for y in reversed(t.order):
        g = grad.pop(y)
        if t.ch[y]:
            a, b = t.sums(p1, y), t.sums(p2, y)
            e = g[:, :, None] * a.exp()
            t.sums(g1, y).copy_(e * (below.pop(y)[:, None, :] + a - b + 1.0))
            t.sums(g2, y).copy_(-e)
            g = e.sum(1)
            grad.update((c, g) for c in t.ch[y])
        d = t.leaf(p1, y) - t.leaf(p2, y)
        t.leaf(g1, y).copy_(g[:, :, None] * (d + 1.0))
        t.leaf(g2, y).copy_(g[:, :, None] * d.exp())     # the sign that the gradient of a leaf is returned with
    return up[t.root][:, 0], g1, g2


def _exact_adam(t, q, p):
    k0, g, _ = _exact_kld(t, q[None], p[None])
    g = g[0]
    b1, b2 = (float(np.float32(1) - np.float32(b)) for b in (0.9, 0.999))     # the rates are float32 arguments
    m, v = b1 * g, b2 * g * g
    q = q - 1e-2 * (m / b1) / ((v / b2).sqrt() + 1e-8)
    for y in t.order:
        for part in ([t.sums(q, y)] if t.ch[y] else []) + [t.leaf(q, y)]:
            part -= torch.logsumexp(part, -1, keepdim=True)
    return {"kld": k0, "q": q, "m": m, "v": v}


def _exact_soft(case, t, p, u):
    key = (p[:, :u.shape[1]] - (-(u * (1.0 - 1e-6) + 1e-6).log()).log()) / 0.7
    out = torch.empty(p.shape[0], case["vars"], case["cats"], dtype=torch.float64, device=p.device)
    prob = {t.root: p.new_ones(p.shape[0], 1)}
    for y in reversed(t.order):
        w = prob.pop(y)
        if t.ch[y]:
            w = (w[:, :, None] * torch.softmax(t.sums(key, y), -1)).sum(1)
            prob.update((c, w) for c in t.ch[y])
        out[:, y] = (w[:, :, None] * t.leaf(p, y).exp()).sum(1)
    return out


def _exact_nflows(case, s, t, theta):
    x = s["data"].t.long()
    kept, _ = t.up(theta, lambda y: t.leaf(theta, y)[:, x[y]].t())
    out = torch.full((theta.numel(), case["batch"]), -math.inf, dtype=torch.float64, device=theta.device)
    eps = float(np.float32(1e-8))
    for y, f, g in t.down(theta, kept):
        if g is not None:
            at, r = t.sum_at[y]
            flow = t.sums(theta, y).exp()[:, :, None] * g.t()[:, None, :] * kept.pop(y)[0].t()[None]
            out[at:at + r * t.k] = (flow / (eps + flow.sum(1, keepdim=True)) + eps).log_().flatten(0, 1)
        at = t.leaf_at[y]
        out[at:at + t.k * t.cats].unflatten(0, (t.k, t.cats)).scatter_(1, x[y].expand(t.k, 1, -1), (f / f).log().t()[:, None])
    return out.t()


def _exact_mi(case, s):
    x = s["data"].t.long()
    v, c, n = case["vars"], case["cats"], case["batch"]
    hot = torch.zeros(v, c, n, device=x.device).scatter_(1, x[:, None], 1.0)     # counts are exact in float32
    total = n + 0.1
    single = ((hot.sum(2).double() + 0.1 / c) / total).log()
    hot = hot.view(v * c, n)
    out = torch.empty(v, v, dtype=torch.float64, device=x.device)
    step = max(1, (1 << 27) // (v * c * c))
    for i in range(0, v, step):
        p = (hot[i * c:(i + step) * c] @ hot.t()).view(-1, c, v, c).double().add_(0.1 / (c * c)).div_(total)
        out[i:i + step] = (p * (p.log() - single[i:i + step, :, None, None] - single)).sum((1, 3))
    return out


def exact(case, seed):
    kind = case["kind"]
    s = prepare(case, seed)
    if kind == "sample":
        return None
    if kind == "mi":
        return _exact_mi(case, s)
    t = _Tree(case)
    if kind == "soft":
        return _exact_soft(case, t, s["params"].double(), s["u"].double())
    if kind == "kld":
        k, g1, g2 = _exact_kld(t, s["p1"].double(), s["p2"].double())
        return {"kld": k, "g1": g1, "g2": g2}
    if kind == "kld_adam":
        return _exact_adam(t, s["q"].double(), s["theta"].double())
    theta = s["theta"].double()
    if kind == "nflows":
        return _exact_nflows(case, s, t, theta)
    if kind == "ll":
        x, miss, out = s["data"].t.long(), s["data"].miss, []
        for r in range(0, case["rows"], 2048):
            def value(y):
                v = t.leaf(theta, y)[:, x[y, r:r + 2048]].t()
                return v if miss is None else v.masked_fill(miss[y, r:r + 2048].bool()[:, None], 0.0)
            out.append(t.up(theta, value)[1])
        return torch.cat(out)
    return _exact_em(case, s, t, theta)


def tolerance(case):
    """Four times what the outputs were measured to be off from the oracle's float64 (training: its float32) results.
    Samples are whole numbers.  A training step on images is the widest: flows are exponentials of differences of
    log-values in the hundreds, whose float32 spacing is up to 6e-5, along a chain of 160 layers."""
    kind = case["kind"]
    if kind == "sample":
        return "exact"
    return {"rel": {"em": 1.3e-4, "em_soft": 1e-5, "ll": 4e-6, "nflows": 2e-6}.get(kind, 1e-6)}
