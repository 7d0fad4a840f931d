"""The work that programs have this engine do, as measurable cases.

Six kinds, each through the package's public entry points (phylommand_gb300.plk):

  eval     one step of a parameter search: a new substitution model on a
           handle that holds an alignment and a tree, then the log-likelihood
           (what treeator's optimiser calls thousands of times);
  whole    the whole call sequence for one alignment and one tree, as treeator
           runs it for every tree and partition: alignment, tree, model, lnL;
  nodes    a new model, its log-likelihood and the normalised state
           probabilities of every internal node;
  batch    one round of many fits at once: the lnL of every alignment of an
           uneven batch at new GTR+Gamma parameters;
  nni      the lnL of every NNI neighbour of every tree of an uneven batch;
  edges    first and second derivatives of lnL in every branch length of every
           tree of an uneven batch (one Newton step of the branch optimiser);
  train    a pass of the warm-start network over a labelled set: minibatch
           Adam steps, then the weights.

Alignments are simulated down a Yule tree on the GPU under the case's own kind
of model, with 2 % missing cells (and, for DNA, 1 % two-state ambiguity codes).
"""
import math
import random

import numpy as np
import torch

from phylommand_gb300 import plk

DEV = "cuda" if torch.cuda.is_available() else "cpu"


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest use: a JC69 tree of 16 taxa in the engine's default
        # arithmetic (the reference's), lnL and ancestral states; latency
        dict(name="nodes_jc_16x1000", kind="nodes", states=4, taxa=16, sites=1000, cats=1, fp64=True, taylor=True,
             marginal=True, bl=0.1),
        # the example alignment's size through the whole call sequence, as the
        # reference's command line runs it (FP64, one category)
        dict(name="whole_dna_103x694", kind="whole", states=4, taxa=103, sites=694, cats=1, fp64=True, taylor=True,
             bl=0.05),
        # the benchmark: a GTR+Gamma4 search step on 128 taxa, 100,000 sites
        dict(name="eval_dna_128x100000", kind="eval", states=4, taxa=128, sites=100000, cats=4, fp64=False,
             taylor=False, persite=False, bl=0.05),
        # a phylogenomic alignment: many taxa, many sites, odd sizes
        dict(name="eval_dna_501x299999", kind="eval", states=4, taxa=501, sites=299999, cats=4, fp64=False,
             taylor=False, persite=False, bl=0.05),
        # proteins, GTR20+Gamma4, the protein benchmark's size
        dict(name="eval_aa_64x20000", kind="eval", states=20, taxa=64, sites=20000, cats=4, fp64=False, taylor=False,
             persite=False, bl=0.1),
        # proteins in the engine's default arithmetic, with per-site values
        dict(name="eval_aa_fp64_40x1501", kind="eval", states=20, taxa=40, sites=1501, cats=4, fp64=True, taylor=True,
             persite=True, bl=0.1),
        # discrete morphological characters: a small alphabet of their own
        dict(name="eval_s5_77x5000", kind="eval", states=5, taxa=77, sites=5000, cats=4, fp64=False, taylor=False,
             persite=True, bl=0.1),
        # ancestral reconstruction of a gene alignment
        dict(name="nodes_dna_100x10000", kind="nodes", states=4, taxa=100, sites=10000, cats=4, fp64=False,
             taylor=False, marginal=True, bl=0.05),
        # uneven batches (taxa 8-256, sites 200-50,000): a fit round, NNI
        # scoring, branch-length derivatives
        dict(name="batch_48", kind="batch", items=48, max_taxa=256, max_sites=50000, cats=4, shapes=1),
        dict(name="nni_48", kind="nni", items=48, max_taxa=256, max_sites=50000, cats=4, shapes=2),
        dict(name="edges_24", kind="edges", items=24, max_taxa=256, max_sites=50000, cats=4, shapes=3),
        # the warm-start network: 16 minibatches of 256
        dict(name="train_16x256", kind="train", steps=16, rows=256, hidden=256, layers=3),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["eval", "eval", "eval", "whole", "nodes", "batch", "nni", "edges", "train"])
    if kind in ("eval", "whole", "nodes"):
        states = rng.choice([4, 4, 4, 20, rng.choice([2, 3, 5, 7, 12, 24])])
        cats = rng.choice([1, 4, 4, 8, 5])
        fp64 = rng.random() < 0.4
        # the cells (taxa x sites x categories x states^2) a kind is used for:
        # FP64 and node states on single genes, FP32 searches up to genomes
        most = {"eval": 2e9, "whole": 5e8, "nodes": 6e7}[kind] / (16.0 if fp64 and kind != "nodes" else 1.0)
        taxa = _log_int(rng, 5, 500 if states == 4 else 128)
        sites = _log_int(rng, 60, max(100, min(300000, int(most / (taxa * cats * states * states)))))
        c = dict(kind=kind, states=states, taxa=taxa, sites=sites, cats=cats, fp64=fp64, taylor=fp64 and rng.random() < 0.7,
                 bl=round(math.exp(rng.uniform(math.log(0.02), math.log(0.2))), 4))
        if kind == "eval":
            c["persite"] = rng.random() < 0.5
        if kind == "nodes":
            c["marginal"] = rng.random() < 0.7
        return c
    if kind == "train":
        return dict(kind=kind, steps=rng.choice([4, 8, 16]), rows=_log_int(rng, 32, 256), hidden=rng.choice([64, 128, 256]),
                    layers=rng.choice([2, 3]))
    cats = rng.choice([1, 4, 4, 8])
    return dict(kind=kind, items=rng.randint(2, 20 if kind == "edges" else 40), max_taxa=rng.choice([32, 100, 256]),
                max_sites=_log_int(rng, 1000, 12000 if cats == 8 else 30000), cats=cats, shapes=rng.randrange(1 << 20))


def _batch_shapes(case):
    """(taxa, sites) of every item: part of the case, not of the seed."""
    r = random.Random(case["shapes"])
    return [(r.randint(8, case["max_taxa"]), _log_int(r, 200, case["max_sites"])) for _ in range(case["items"])]


# ------------------------------------------------------------------ the inputs
def _yule(n, mean_bl, rng):
    """Random joins of two lineages: tips 0..n-1, internal nodes in creation
    order, the root last; exponential branch lengths."""
    m = 2 * n - 1
    left, right = np.full(m, -1, dtype=np.int32), np.full(m, -1, dtype=np.int32)
    lineages = list(range(n))
    for v in range(n, m):
        i, j = rng.choice(len(lineages), size=2, replace=False)
        left[v], right[v] = lineages[i], lineages[j]
        for q in sorted((int(i), int(j)), reverse=True):
            lineages.pop(q)
        lineages.append(v)
    bl = rng.exponential(mean_bl, size=m) + 1e-6
    bl[m - 1] = 0.0
    return left, right, bl


def _gamma_rates(alpha, K):
    """Mean rates of K equal-probability categories of a mean-1 Gamma (Yang
    1994), quantiles by bisection on the regularised incomplete gamma."""
    if K == 1:
        return np.ones(1)
    a = torch.tensor(alpha, dtype=torch.float64)
    p = torch.arange(1, K, dtype=torch.float64) / K
    lo, hi = torch.zeros(K - 1, dtype=torch.float64), torch.full((K - 1,), 2000.0 * (1 + alpha), dtype=torch.float64)
    for _ in range(200):
        mid = 0.5 * (lo + hi)
        up = torch.special.gammainc(a, mid) < p
        lo, hi = torch.where(up, mid, lo), torch.where(up, hi, mid)
    cdf = torch.special.gammainc(a + 1, 0.5 * (lo + hi)).numpy()
    return K * np.diff(np.concatenate(([0.0], cdf, [1.0])))


def _gtr(exch, freqs):
    """Reversible Q of mean rate 1."""
    S = len(freqs)
    Q = np.zeros((S, S))
    Q[np.triu_indices(S, 1)] = exch
    Q = (Q + Q.T) * freqs[None, :]
    np.fill_diagonal(Q, -Q.sum(axis=1))
    return Q / -float(np.dot(freqs, np.diag(Q)))


def _model(case, rng):
    S, C = case["states"], case["cats"]
    npos = S * (S - 1) // 2
    if S == 4 and C == 1 and case.get("taylor"):
        return np.full((4, 4), 1.0 / 3.0) - np.eye(4) * (4.0 / 3.0), np.full(4, 0.25), np.ones(1), np.ones(1)  # JC69
    exch = rng.lognormal(0.0, 1.0, npos) if S == 20 else rng.uniform(0.5, 5.0, npos)
    freqs = rng.dirichlet(np.full(S, 5.0 if S == 20 else 10.0))
    return _gtr(exch, freqs), freqs, _gamma_rates(float(rng.uniform(0.4, 1.2)), C), np.full(C, 1.0 / C)


def _simulate(left, right, bl, Q, freqs, rates, sites, gen):
    """State sets [taxa, sites] (int32, on the GPU) simulated down the tree."""
    S, C, m = len(freqs), len(rates), len(left)
    n = (m + 1) // 2
    q = torch.from_numpy(Q)
    t = torch.from_numpy(bl[:, None] * np.asarray(rates)[None, :])
    P = torch.linalg.matrix_exp(q[None, None] * t[:, :, None, None]).clamp_min(0)
    cum = (P / P.sum(-1, keepdim=True)).cumsum(-1)[..., :-1].contiguous().float().to(DEV)  # [m, C, S, S - 1]
    row = torch.randint(0, C, (sites,), generator=gen, device=DEV) * S
    state = {m - 1: torch.multinomial(torch.from_numpy(freqs).float().to(DEV), sites, replacement=True, generator=gen)}
    out = torch.empty((n, sites), dtype=torch.int32, device=DEV)
    for u in range(m - 1, n - 1, -1):
        base = row + state.pop(u)
        for v in (int(left[u]), int(right[u])):
            edges = cum[v].reshape(C * S, S - 1).index_select(0, base)
            s = (torch.rand((sites, 1), generator=gen, device=DEV) >= edges).sum(1)
            if v < n:
                out[v] = torch.ones_like(s, dtype=torch.int32) << s
            else:
                state[v] = s
    u = torch.rand((n, sites), generator=gen, device=DEV)
    out[u < 0.02] = (1 << S) - 1
    if S == 4:  # purine / pyrimidine codes
        amb = (u >= 0.02) & (u < 0.03)
        out[amb] = torch.where((out[amb] & 3) != 0, 3, 12).to(torch.int32)
    return out


def _single(case, seed):
    """Tree, model and state sets of a one-alignment case, from the seed."""
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=DEV).manual_seed(seed)
    left, right, bl = _yule(case["taxa"], case["bl"], rng)
    Q, freqs, rates, weights = _model(case, rng)
    masks = _simulate(left, right, bl, Q, freqs, rates, case["sites"], gen)
    return left, right, bl, Q, freqs, rates, weights, masks


def _host_masks(masks, S):
    """As a program holds them: bytes for DNA, 32-bit sets for other alphabets."""
    return masks.to(torch.uint8).cpu().numpy() if S == 4 else masks.cpu().numpy().astype(np.uint32)


def _batch(case, seed):
    """Per item of a batch: tree, state sets, frequencies, fit parameters."""
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=DEV).manual_seed(seed)
    items = []
    for taxa, sites in _batch_shapes(case):
        left, right, bl = _yule(taxa, 0.05, rng)
        x = np.concatenate([np.log(rng.uniform(0.5, 2.0, 5)), np.log(rng.uniform(0.3, 2.0, 1 if case["cats"] > 1 else 0)),
                            rng.normal(0.0, 0.1, 1)])
        freqs = rng.dirichlet(np.full(4, 10.0))
        Q, rates = _gtr_point(x, freqs, case["cats"])
        masks = _simulate(left, right, bl, Q, freqs, rates, sites, gen)
        items.append((left, right, bl, x, freqs, Q, rates, masks))
    return items


def _gtr_point(x, freqs, C):
    """The model at a fit's parameter vector: log exchangeabilities relative to
    the last one, log alpha (two or more categories), log tree-length scale."""
    Q = _gtr(np.concatenate([np.exp(x[:5]), [1.0]]), freqs)
    return Q, _gamma_rates(float(np.exp(x[5])), C) * float(np.exp(x[-1]))


def _network(case, seed):
    """Initial weights, standardised features and labels of a training pass."""
    rng = np.random.default_rng(seed)
    n = case["steps"] * case["rows"]
    x = rng.normal(size=(n, 43)).astype(np.float32)
    mix = rng.normal(size=(43, 7)) / math.sqrt(43)
    t = (np.tanh(x @ mix) + 0.1 * rng.normal(size=(n, 7))).astype(np.float32)
    dims = [43] + [case["hidden"]] * case["layers"] + [7]
    p = [np.concatenate([(rng.normal(size=(b, a)) * math.sqrt(2.0 / a)).ravel(), np.zeros(b)]) for a, b in zip(dims, dims[1:])]
    return dims, np.concatenate(p).astype(np.float32), x, t


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        dims, p, x, t = _network(case, seed)
        net = plk.MLP(43, 7, case["hidden"], case["layers"], seed=seed)
        net.set_params(p)
        r = case["rows"]
        return dict(kind=kind, net=net, data=[(x[i * r:(i + 1) * r], t[i * r:(i + 1) * r]) for i in range(case["steps"])])
    if kind in ("batch", "nni", "edges"):
        b = plk.Batch(case["cats"])
        items = _batch(case, seed)
        for left, right, bl, x, freqs, Q, rates, masks in items:
            i = b.add(masks.cpu().numpy().astype(np.uint32), left, right, bl)
            b.set_model(i, Q, freqs, rates, np.full(case["cats"], 1.0 / case["cats"]))
        return dict(kind=kind, batch=b, freqs=np.stack([it[4] for it in items]), x=np.stack([it[3] for it in items]))
    left, right, bl, Q, freqs, rates, weights, masks = _single(case, seed)
    S = case["states"]
    h = plk.Handle()
    st = dict(kind=kind, h=h, S=S, masks=_host_masks(masks, S), tree=(left, right, bl),
              model=(Q, freqs, True, rates, weights, plk.PLK_P_TAYLOR20 if case["taylor"] else plk.PLK_P_EXACT),
              precision=plk.PLK_FP64 if case["fp64"] else plk.PLK_FP32S, persite=case.get("persite", False),
              mode=plk.PLK_NODES_MARGINAL if case.get("marginal") else plk.PLK_NODES_COND)
    if kind != "whole":
        h.set_alignment(st["masks"], S)
        h.set_tree(left, right, bl)
        h.set_rate_model(False)
    return st


def run(st):
    kind = st["kind"]
    if kind == "train":
        return dict(loss=[st["net"].train_step(x, t, 1e-3) for x, t in st["data"]], weights=st["net"].get_params())
    if kind == "batch":
        return st["batch"].eval_gtr(st["freqs"], st["x"])
    if kind == "nni":
        return st["batch"].nni_loglik()
    if kind == "edges":
        return st["batch"].edge_derivatives()
    h = st["h"]
    if kind == "whole":
        h.set_alignment(st["masks"], st["S"])
        h.set_tree(*st["tree"])
        h.set_rate_model(False)
    h.set_model(*st["model"])
    out = dict(lnl=h.loglik(st["precision"]))
    if st["persite"]:
        out["site"] = h.site_loglik()
    if kind == "nodes":
        out["nodes"] = h.node_states(st["mode"], st["precision"])
    return out


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    """Bytes: the tip state sets (one byte a cell; for "whole" as the caller
    holds them) and the outputs; flops: the products of every internal child's
    vector with P(t) and the combines (tips are look-ups)."""
    kind = case["kind"]
    if kind == "train":
        dims = [43] + [case["hidden"]] * case["layers"] + [7]
        nw = sum(a * b for a, b in zip(dims, dims[1:]))
        n = case["steps"] * case["rows"]
        return {"bytes": 4.0 * (n * 50 + 8 * nw * case["steps"]), "flops": 6.0 * nw * n}
    if kind in ("batch", "nni", "edges"):
        C, by, fl = case["cats"], 0.0, 0.0
        for n, N in _batch_shapes(case):
            by += n * N + 8 * (2 * (n - 3) if kind == "nni" else 2 * (2 * n - 1) if kind == "edges" else 1)
            post = ((n - 2) * 2 * C * 16 + (n - 1) * C * 4) * N
            # pre-order: one transposed product and two combines per internal edge
            pre = (n - 2) * C * (32 + 8) * N
            # a move: two combines, one product, the root sum
            moves = 2 * (n - 3) * C * (32 + 4 + 4 + 9) * N
            # an edge: both eigen projections (two products) and three sums
            edges = (2 * n - 2) * C * (64 + 4 + 24) * N
            fl += post + (pre + moves if kind == "nni" else pre + edges if kind == "edges" else 0)
        return {"bytes": by, "flops": fl}
    S, C, n, N = case["states"], case["cats"], case["taxa"], case["sites"]
    by = float(n * N) * (4 if kind == "whole" and S != 4 else 1) + 8
    fl = float(N) * ((n - 2) * 2 * C * S * S + (n - 1) * C * S)
    if case.get("persite"):
        by += 8 * N
    if kind == "nodes":
        by += 8.0 * (n - 1) * N * S
        # the mix over categories; marginal: an outside vector per internal
        # node (a transposed product, its sibling's message) and the mix
        fl += float(N) * (n - 1) * C * S * 2 + (float(N) * (n - 2) * C * (4 * S * S + 2 * S) if case["marginal"] else 0.0)
    return {"bytes": by, "flops": fl}


# ------------------------------------------------------------------ the same in 64 bits
def _pmats(Q, t, rates, taylor):
    """P [nodes, C, S, S] on the GPU: exp(Q t r), or (I + Q t r / 2^20)^(2^20)."""
    A = torch.from_numpy(Q)[None, None] * torch.from_numpy(t[:, None] * np.asarray(rates)[None, :])[:, :, None, None]
    if taylor:
        P = torch.eye(len(Q), dtype=torch.float64) + A / 1048576.0
        for _ in range(20):
            P = P @ P
    else:
        P = torch.linalg.matrix_exp(A)
    return P.to(DEV)


def _times(x, P):
    """out[k, n, i] = sum_j P[k, i, j] x[k, n, j]."""
    return torch.matmul(x, P.transpose(1, 2))


def _postorder(left, right, root):
    order, stack = [], [(root, False)]
    while stack:
        v, seen = stack.pop()
        if left[v] < 0:
            continue
        if seen:
            order.append(v)
        else:
            stack += [(v, True), (int(right[v]), False), (int(left[v]), False)]
    return order


class _Tree64:
    """Conditional vectors, messages to the parent and outside vectors of one
    alignment in 64 bits, each scaled per site (logs of the scales beside)."""

    def __init__(self, left, right, P, sets, freqs, S, keep, outside):
        n, m = (len(left) + 1) // 2, len(left)
        self.root, self.P, C = m - 1, P, P.shape[1]
        self.order = _postorder(left, right, m - 1)
        bits = (sets[:, :, None] >> torch.arange(S, device=DEV, dtype=torch.int32)) & 1
        self.cond, self.D, self.sc = {}, {}, {}
        one = torch.zeros(sets.shape[1], dtype=torch.float64, device=DEV)
        for v in range(n):
            tip = bits[v].double()[None].expand(C, -1, -1)
            self.cond[v], self.sc[v] = tip, one
            self.D[v] = _times(tip, P[v])
        for u in self.order:
            a, b = int(left[u]), int(right[u])
            x = self.D[a] * self.D[b]
            mx = x.amax((0, 2))
            self.cond[u], self.sc[u] = x / mx[None, :, None], self.sc[a] + self.sc[b] + torch.log(mx)
            if u != m - 1:
                self.D[u] = _times(self.cond[u], P[u])
            if not keep:
                for v in (a, b):
                    del self.D[v], self.cond[v], self.sc[v]
        if outside:
            pi = torch.from_numpy(freqs).to(DEV)
            self.O = {m - 1: pi[None, None, :].expand(C, sets.shape[1], S)}
            self.osc = {m - 1: one}
            for u in reversed(self.order):
                for v, w in ((int(left[u]), int(right[u])), (int(right[u]), int(left[u]))):
                    if v < n:
                        continue
                    o = torch.matmul(self.O[u] * self.D[w], P[v])
                    mx = o.amax((0, 2))
                    self.O[v] = o / mx[None, :, None]
                    self.osc[v] = self.osc[u] + self.sc[w] + torch.log(mx)


def _mix(x, weights):
    return torch.einsum("k,kn->n", torch.from_numpy(np.asarray(weights, dtype=np.float64)).to(DEV), x)


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_train(case, seed)
    if kind in ("batch", "nni", "edges"):
        return _exact_batch(case, seed)
    left, right, bl, Q, freqs, rates, weights, masks = _single(case, seed)
    S, n, N = case["states"], case["taxa"], case["sites"]
    P = _pmats(Q, bl, rates, case["taylor"])
    pi = torch.from_numpy(freqs).to(DEV)
    nodes = kind == "nodes"
    step = max(1, int(2e7 / (case["cats"] * S * (2 * n if nodes else 8))))
    site, states = [], []
    for s in range(0, N, step):
        t = _Tree64(left, right, P, masks[:, s:s + step], freqs, S, nodes, nodes and case["marginal"])
        site.append(torch.log(_mix(t.cond[t.root] @ pi, weights)) + t.sc[t.root])
        if nodes:
            w = torch.from_numpy(weights).to(DEV)
            rows = []
            for u in t.order:
                x = t.cond[u] * t.O[u] if case["marginal"] else t.cond[u]
                x = torch.einsum("k,kns->ns", w, x)
                rows.append(x / x.sum(1, keepdim=True))
            states.append(torch.stack(rows).cpu())
    site = torch.cat(site)
    out = dict(lnl=float(site.sum()))
    if case.get("persite"):
        out["site"] = site.cpu().numpy()
    if nodes:
        out["nodes"] = torch.cat(states, 1).numpy()
    return out


def _exact_batch(case, seed):
    kind, C = case["kind"], case["cats"]
    weights = np.full(C, 1.0 / C)
    got = []
    for left, right, bl, x, freqs, Q, rates, masks in _batch(case, seed):
        P = _pmats(Q, bl, rates, False)
        pi = torch.from_numpy(freqs).to(DEV)
        n, m = (len(left) + 1) // 2, len(left)
        t = _Tree64(left, right, P, masks, freqs, 4, kind != "batch", kind != "batch")
        if kind == "batch":
            got.append(float((torch.log(_mix(t.cond[t.root] @ pi, weights)) + t.sc[t.root]).sum()))
            continue
        parent = {int(c): u for u in range(n, m) for c in (left[u], right[u])}

        def total(lk, *scales):
            return float((torch.log(_mix(lk, weights)) + sum(scales)).sum())

        if kind == "nni":
            moves = []
            for v in t.order:
                if v == t.root:
                    continue
                u = parent[v]
                c = int(right[u]) if left[u] == v else int(left[u])
                a, b = int(left[v]), int(right[v])
                if u != t.root:
                    for x1, y1, z1 in ((a, c, b), (c, b, a)):
                        vec = _times(t.D[x1] * t.D[y1], P[v])
                        moves.append(total((t.O[u] * vec * t.D[z1]).sum(2), t.sc[a], t.sc[b], t.sc[c], t.osc[u]))
                elif left[u] == v and c >= n:
                    d, e = int(left[c]), int(right[c])
                    for x1, y1, p1, q1 in ((a, d, b, e), (a, e, d, b)):
                        vec = _times(t.D[x1] * t.D[y1], P[v]) * _times(t.D[p1] * t.D[q1], P[c])
                        moves.append(total(vec @ pi, t.sc[a], t.sc[b], t.sc[d], t.sc[e]))
            got.append(np.array(moves))
        else:
            d = np.zeros((m, 2))
            q = torch.from_numpy(Q).to(DEV)
            r = torch.from_numpy(np.asarray(rates)).to(DEV)[:, None, None]
            for u in t.order:
                for v, w in ((int(left[u]), int(right[u])), (int(right[u]), int(left[u]))):
                    A = t.O[u] * t.D[w]
                    P1 = r * torch.matmul(q, P[v])
                    P2 = r * torch.matmul(q, P1)
                    l0, l1, l2 = (_mix((A * _times(t.cond[v], M)).sum(2), weights) for M in (P[v], P1, P2))
                    g = l1 / l0
                    d[v] = float(g.sum()), float((l2 / l0 - g * g).sum())
            got.append(d)
    return np.array(got) if kind == "batch" else got


def _exact_train(case, seed):
    dims, p, x, t = _network(case, seed)
    w = torch.from_numpy(p).double().requires_grad_(True)
    opt = torch.optim.Adam([w], lr=1e-3, betas=(0.9, 0.999), eps=1e-8)
    losses, r = [], case["rows"]
    for i in range(case["steps"]):
        a, off = torch.from_numpy(x[i * r:(i + 1) * r]).double(), 0
        for l, (k, m) in enumerate(zip(dims, dims[1:])):
            a = a @ w[off:off + k * m].reshape(m, k).T + w[off + k * m:off + k * m + m]
            off += k * m + m
            a = torch.relu(a) if l + 2 < len(dims) else a
        loss = ((a - torch.from_numpy(t[i * r:(i + 1) * r]).double()) ** 2).mean()
        opt.zero_grad()
        loss.backward()
        opt.step()
        losses.append(float(loss))
    return dict(loss=losses, weights=w.detach().numpy())
