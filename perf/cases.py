"""Performance cases of the pruning likelihood: what a program built on this
package has it do, over the range of sizes it is used at.

Kinds of case:

  proposals  a maximum-likelihood or MCMC driver proposes model parameters on
             one tree (new exchangeabilities, then a new Gamma shape, ...) and
             asks for the lnL of each: every proposal recomputes every node.
  branches   the same driver proposes single branch lengths: each recomputes
             the path from the branch to the root.
  sites      the lnL of every site of an alignment as read (not compacted)
             after a model change, through the drop-in entry point on host CL
             structs (plain FP64).
  batch      many (tree, alignment) jobs of uneven size in one launch.
  mc3        generations of on-device Metropolis-coupled chains.
  serve      a burst of lnL requests of uneven size to the serving loop, on
             alignments kept resident.
  compact    pattern compression of a raw host alignment on the device.

Trees are Yule trees with exponential branch lengths and sequences are
simulated on them under GTR with discrete Gamma rates, optional invariant
sites and 0.5 % gaps, which is what the tests and the benchmark use.
"""
import math

import numpy as np
import torch

from crux_gb300 import Alignment, Lik, TaxaMap, Tree
from crux_gb300.batch import Batch
from crux_gb300.compact import compact, compact_alignment
from crux_gb300.mc3 import Mc3
from crux_gb300.serve import PreparedRequest, Server
from crux_gb300.synth import apply_params

CODES = np.frombuffer(b"ACGT-", dtype=np.uint8)

# Most taxa x sites a drawn case of each kind may have.
LARGEST = {"proposals": 128 * 100000, "branches": 128 * 100000,
           "sites": 96 * 30000, "mc3": 128 * 50000,
           "compact": 128 * 100000}


def listed():
    return [
        # The smallest call of the plain form: launches and host work count.
        {"name": "proposals_fp64_16x1000", "kind": "proposals", "taxa": 16, "sites": 1000,
         "precision": "fp64", "ncat": 4, "pinv": 0.0, "models": 1, "brlen": 0.1, "n": 8},
        # Branch-length proposals on a mid-size tree with invariant sites
        # (five components): a few nodes per call.
        {"name": "branches_fp32_64x10000_inv", "kind": "branches", "taxa": 64, "sites": 10000,
         "precision": "fp32", "ncat": 4, "pinv": 0.2, "models": 1, "brlen": 0.05, "n": 16},
        # The same on a large alignment in the plain form.
        {"name": "branches_fp64_128x60000", "kind": "branches", "taxa": 128, "sites": 60000,
         "precision": "fp64", "ncat": 4, "pinv": 0.0, "models": 1, "brlen": 0.05, "n": 8},
        # The benchmark's workload: model proposals on 128 taxa x 100,000
        # sites, in the FP32 form and in the plain form.
        {"name": "proposals_fp32_128x100000", "kind": "proposals", "taxa": 128, "sites": 100000,
         "precision": "fp32", "ncat": 4, "pinv": 0.0, "models": 1, "brlen": 0.05, "n": 8},
        {"name": "proposals_fp64_128x100000", "kind": "proposals", "taxa": 128, "sites": 100000,
         "precision": "fp64", "ncat": 4, "pinv": 0.0, "models": 1, "brlen": 0.05, "n": 4},
        # A mixture of two models with Gamma rates (eight components), odd sizes.
        {"name": "proposals_fp32_41x30011_mix2", "kind": "proposals", "taxa": 41, "sites": 30011,
         "precision": "fp32", "ncat": 4, "pinv": 0.0, "models": 2, "brlen": 0.05, "n": 8},
        # One rate category on many taxa and few sites (a gene alignment).
        {"name": "proposals_fp32_509x5003_nogamma", "kind": "proposals", "taxa": 509, "sites": 5003,
         "precision": "fp32", "ncat": 1, "pinv": 0.0, "models": 1, "brlen": 0.05, "n": 8},
        # Per-site lnLs through the drop-in entry point.
        {"name": "sites_dropin_48x20011", "kind": "sites", "taxa": 48, "sites": 20011,
         "precision": "fp64", "ncat": 4, "pinv": 0.0, "models": 1, "brlen": 0.05, "n": 2},
        # Uneven jobs (16-512 taxa, 500-50,000 sites) in one launch.
        {"name": "batch_fp32_32jobs", "kind": "batch", "jobs": 32, "taxa_lo": 16, "taxa_hi": 512,
         "sites_lo": 500, "sites_hi": 50000, "precision": "fp32", "ncat": 4, "brlen": 0.05},
        # On-device MC3 on a large alignment: eight chains, branch-length,
        # topology and model moves.
        {"name": "mc3_fp32_128x50000_8chains", "kind": "mc3", "taxa": 128, "sites": 50000,
         "precision": "fp32", "ncat": 4, "chains": 8, "gens": 32, "brlen": 0.05},
        # A burst of requests to the serving loop.
        {"name": "serve_fp32_24requests", "kind": "serve", "datasets": 6, "requests": 24,
         "taxa_lo": 8, "taxa_hi": 512, "sites_lo": 200, "sites_hi": 50000,
         "precision": "fp32", "ncat": 4, "brlen": 0.05},
        # Pattern compression of a raw alignment, host to host.
        {"name": "compact_128x100000", "kind": "compact", "taxa": 128, "sites": 100000,
         "brlen": 0.05},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same kinds, sizes spread over their logarithm."""
    kind = rng.choice(["proposals", "proposals", "proposals", "branches", "branches", "sites",
                       "batch", "mc3", "serve", "compact"])
    brlen = rng.choice([0.05, 0.1])
    prec = rng.choice(["fp32", "fp32", "fp64"])
    if kind == "batch":
        return {"kind": kind, "jobs": _log_int(rng, 4, 32), "taxa_lo": _log_int(rng, 8, 24),
                "taxa_hi": _log_int(rng, 64, 256), "sites_lo": _log_int(rng, 200, 1000),
                "sites_hi": _log_int(rng, 5000, 40000), "precision": prec,
                "ncat": rng.choice([1, 4]), "brlen": brlen}
    if kind == "serve":
        return {"kind": kind, "datasets": rng.randint(2, 6), "requests": rng.randint(8, 24),
                "taxa_lo": 8, "taxa_hi": _log_int(rng, 64, 512), "sites_lo": 200,
                "sites_hi": _log_int(rng, 2000, 50000), "precision": prec, "ncat": 4,
                "brlen": brlen}
    top = LARGEST[kind]
    if kind == "mc3":
        taxa, sites = _log_int(rng, 8, 128), _log_int(rng, 500, 50000)
        return {"kind": kind, "taxa": taxa, "sites": min(sites, top // taxa),
                "precision": "fp32", "ncat": rng.choice([1, 4]),
                "chains": rng.randint(2, 8), "gens": rng.randint(16, 32), "brlen": brlen}
    taxa = _log_int(rng, 8, 512)
    sites = min(_log_int(rng, 200, 100000), top // taxa)
    if kind == "compact":
        return {"kind": kind, "taxa": taxa, "sites": sites, "brlen": brlen}
    ncat = rng.choice([1, 4, 4, 4])
    models = 2 if ncat == 4 and rng.random() < 0.2 else 1
    pinv = rng.choice([0.0, 0.0, 0.2]) if models == 1 else 0.0
    n = {"proposals": 4, "branches": 8, "sites": 2}[kind]
    return {"kind": kind, "taxa": taxa, "sites": sites,
            "precision": "fp64" if kind == "sites" else prec, "ncat": ncat, "pinv": pinv,
            "models": models, "brlen": brlen, "n": n}


# -- inputs -------------------------------------------------------------------

class Data:
    """One simulated alignment with its tree, as plain arrays: a rooted Yule
    tree (children lists, a length above every node, leaves in taxon order)
    and the leaves' states [taxa][sites] (4: gap)."""

    def __init__(self, taxa, sites, rng, ncat=4, pinv=0.0, models=1, brlen=0.05):
        kids, leaves, nxt = {0: ()}, [0], 1
        while len(leaves) < taxa:
            i = int(rng.integers(len(leaves)))
            v = leaves[i]
            kids[v], kids[nxt], kids[nxt + 1] = (nxt, nxt + 1), (), ()
            leaves[i] = nxt
            leaves.append(nxt + 1)
            nxt += 2
        self.taxa, self.sites, self.ncat, self.pinv = taxa, sites, ncat, pinv
        self.kids = [kids[v] for v in range(nxt)]
        self.leaf = {v: i for i, v in enumerate(sorted(leaves))}
        self.len = rng.exponential(brlen, nxt)
        self.names = ["T%d" % i for i in range(taxa)]
        # Model parameters: one dict per mixture member.
        self.models = [{"rates": [float(x) for x in rng.dirichlet(np.ones(6)) * 6.0],
                        "freqs": [float(x) for x in rng.dirichlet(np.full(4, 5.0))]}
                       for _ in range(models)]
        self.weights = [1.0] + [0.5] * (models - 1)
        self.alpha = float(rng.uniform(0.3, 1.0)) if ncat > 1 else None
        self.seed = int(rng.integers(1 << 40))
        self._states = None

    def order(self):
        """Nodes, parents first."""
        out, stack = [], [0]
        while stack:
            v = stack.pop()
            out.append(v)
            stack.extend(self.kids[v])
        return out

    def newick(self):
        text = {}
        for v in reversed(self.order()):
            me = "(" + ",".join(text[c] for c in self.kids[v]) + ")" if self.kids[v] \
                else self.names[self.leaf[v]]
            text[v] = me if v == 0 else "%s:%r" % (me, float(self.len[v]))
        return text[0] + ";"

    def states(self):
        if self._states is None:
            self._states = self._simulate()
        return self._states

    def _simulate(self):
        dev = "cuda"
        g = torch.Generator(device=dev)
        g.manual_seed(self.seed)
        n = self.sites
        m = self.models[0]
        rates = gamma_means(self.alpha, self.ncat) if self.alpha else [1.0]
        rates = [r / (1.0 - self.pinv) for r in rates] + [0.0]
        cat = torch.randint(len(rates) - 1, (n,), generator=g, device=dev)
        inv = torch.rand(n, generator=g, device=dev) < self.pinv
        cat = torch.where(inv, len(rates) - 1, cat)
        lam, V, W, pi = eigen(m)
        lam = lam / -(pi * rate_matrix(m).diagonal()).sum()
        t = self.len[:, None, None, None, None] * np.array(rates)[None, :, None, None, None]
        P = (V * np.exp(lam * t[..., 0])) @ W                 # [nodes, rates, 4, 4]
        cdf = torch.tensor(np.cumsum(P, -1)[..., :3], dtype=torch.float32, device=dev)
        start = torch.tensor(np.cumsum(pi)[:3], dtype=torch.float32, device=dev)
        state = {0: (torch.rand(n, 1, generator=g, device=dev) > start).sum(1)}
        out = np.zeros((self.taxa, n), dtype=np.uint8)
        for v in self.order():
            if v:
                row = cdf[v][cat, state[self.up[v]]]
                state[v] = (torch.rand(n, 1, generator=g, device=dev) > row).sum(1)
            if not self.kids[v]:
                gap = torch.rand(n, generator=g, device=dev) < 0.005
                out[self.leaf[v]] = torch.where(gap, 4, state[v]).to(torch.uint8).cpu().numpy()
        return out

    @property
    def up(self):
        if not hasattr(self, "_up"):
            self._up = {c: v for v, ks in enumerate(self.kids) for c in ks}
        return self._up

    # For PreparedRequest, which takes its tree and model from a case.
    @property
    def params(self):
        return self.models[0]

    def raw_alignment(self):
        return Alignment(taxaMap=TaxaMap(self.names), rows=CODES[self.states()])

    def alignment(self):
        a = self.raw_alignment()
        compact_alignment(a)
        return a

    def tree(self, taxaMap):
        t = Tree(self.newick())
        t.deroot()
        t.canonize(taxaMap)
        return t

    def lik(self, precision, dropin=False):
        a = self.raw_alignment() if dropin else self.alignment()
        k = Lik(self.tree(a.taxaMap), a, nmodels=len(self.models), ncat=self.ncat,
                invar=self.pinv > 0.0, precision=precision, dropin=dropin)
        for i, m in enumerate(self.models):
            apply_params(k, i, m, self.alpha, self.pinv)
            k.setWeight(i, self.weights[i])
        return k


def _data(case, seed):
    rng = np.random.default_rng([seed, 11])
    d = Data(case["taxa"], case["sites"], rng, ncat=case.get("ncat", 4),
             pinv=case.get("pinv", 0.0), models=case.get("models", 1), brlen=case["brlen"])
    return d, rng


def _jobs(case, seed):
    """The uneven jobs of a batch."""
    out = []
    for j in range(case["jobs"]):
        rng = np.random.default_rng([seed, 13, j])
        taxa, sites = _spread(case, j, case["jobs"])
        out.append(Data(taxa, sites, rng, ncat=case["ncat"], brlen=case["brlen"]))
    return out


def _spread(case, j, n):
    """Size j of n: taxa and sites each cover their range evenly in the
    logarithm, in unrelated orders."""
    a, b = (j * 0.6180339887) % 1.0, (j + 0.5) / n
    return tuple(int(round(lo * (hi / lo) ** f)) for lo, hi, f in
                 ((case["taxa_lo"], case["taxa_hi"], a), (case["sites_lo"], case["sites_hi"], b)))


def _requests(case, seed):
    """The datasets and, per request, (dataset, its own tree lengths, model)."""
    sets = []
    for j in range(case["datasets"]):
        rng = np.random.default_rng([seed, 17, j])
        taxa, sites = _spread(case, j, case["datasets"])
        sets.append(Data(taxa, sites, rng, ncat=case["ncat"], brlen=case["brlen"]))
    rng = np.random.default_rng([seed, 19])
    reqs = []
    for i in range(case["requests"]):
        d = sets[i % len(sets)]
        r = Data.__new__(Data)
        r.__dict__.update(d.__dict__)
        r.len = d.len * rng.uniform(0.8, 1.25, len(d.len))
        r.models = [_jump(d.models[0], rng)]
        reqs.append((i % len(sets), r))
    return sets, reqs


def _jump(m, rng):
    return {"rates": [float(x) for x in np.array(m["rates"]) * np.exp(rng.normal(0, 0.1, 6))],
            "freqs": list(m["freqs"])}


def _proposals(d, rng, n):
    """Model proposals one after another: new exchangeabilities of the first
    model, or (every other time, with Gamma rates) a new shape."""
    out = []
    for i in range(n):
        if i % 2 and d.alpha is not None:
            out.append(("alpha", float(d.alpha * math.exp(rng.normal(0, 0.1)))))
        else:
            out.append(("rates", _jump(d.models[0], rng)["rates"]))
    return out


def _branches(d, rng, n):
    """Leaf branches to rescale, and by how much."""
    at = rng.choice(d.taxa, size=n, replace=n > d.taxa)
    return [(int(i), float(f)) for i, f in zip(at, rng.uniform(0.5, 2.0, n))]


def _repeated(states, rng):
    """`states` with a known number of distinct columns, three in five: those
    differ in the last taxa, which count them, and the others repeat them."""
    taxa, sites = states.shape
    digits = min(taxa, 10)
    distinct = max(1, min(3 * sites // 5, 4 ** digits // 2))
    out = states.copy()
    number = rng.choice(4 ** digits, size=distinct, replace=False)
    for k in range(digits):
        out[taxa - 1 - k, :distinct] = number // 4 ** k % 4
    at = rng.permutation(sites)
    source = np.concatenate([np.arange(distinct),
                             rng.integers(distinct, size=sites - distinct)])
    return np.ascontiguousarray(out[:, source[at]])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        liks = [d.lik(case["precision"]) for d in _jobs(case, seed)]
        for k in liks:
            k.prepare_plan()
        return {"kind": kind, "liks": liks, "batch": Batch(liks, case["precision"])}
    if kind == "serve":
        sets, reqs = _requests(case, seed)
        server = Server(case["precision"], hbm_budget=32 << 30)
        alns = [d.alignment() for d in sets]
        for j, d in enumerate(sets):
            server.add_dataset(j + 1, PreparedRequest(d, alignment=alns[j]))
        return {"kind": kind, "server": server,
                "requests": [PreparedRequest(r, alignment=alns[j], dataset=j + 1)
                             for j, r in reqs]}
    d, rng = _data(case, seed)
    if kind == "compact":
        a = Alignment(taxaMap=TaxaMap(d.names), rows=CODES[_repeated(d.states(), rng)])
        return {"kind": kind, "alignment": a}
    if kind == "mc3":
        a = d.alignment()
        m = Mc3(d.tree(a.taxaMap), a, d.models[0]["rates"], d.models[0]["freqs"], alpha=d.alpha,
                ncat=case["ncat"], nchains=case["chains"], heat_delta=0.1, seed=seed + 1,
                moves=_moves(case), precision=case["precision"])
        return {"kind": kind, "mc3": m, "gens": case["gens"], "chains": case["chains"]}
    lik = d.lik(case["precision"], dropin=kind == "sites")
    s = {"kind": kind, "lik": lik}
    if kind == "branches":
        edge = {}
        for e in lik.tree.edges:
            for ring in (e.ring, e.ring.other):
                if ring.node.taxon is not None:
                    edge[ring.node.taxon] = e
        s["moves"] = [(edge["T%d" % i], f) for i, f in _branches(d, rng, case["n"])]
        lik.lnL()
    else:
        s["proposals"] = _proposals(d, rng, case["n"])
        s["back"] = [("rates", d.models[0]["rates"])]
        if d.alpha is not None:
            s["back"].append(("alpha", d.alpha))
    return s


def _moves(case):
    moves = {"brlen": 2.0, "nni": 1.0, "spr": 1.0, "rates": 1.0}
    if case["ncat"] > 1:
        moves["alpha"] = 1.0
    return moves


def _propose(lik, what, value):
    if what == "alpha":
        for m in range(lik.nmodels()):
            lik.setAlpha(m, value)
    else:
        lik.setRclass(0, [0, 1, 2, 3, 4, 5], value)


def _back(state):
    """The proposals are rejected: the model is what it was."""
    for what, value in state["back"]:
        _propose(state["lik"], what, value)


def run(state):
    kind = state["kind"]
    if kind == "proposals":
        lik, out = state["lik"], []
        for what, value in state["proposals"]:
            _propose(lik, what, value)
            out.append(lik.lnL())
        _back(state)
        return np.array(out)
    if kind == "branches":
        # Each branch is rescaled, evaluated and (the proposals rejected, last
        # first) put back and evaluated again.
        lik, out, old = state["lik"], [], []
        for edge, f in state["moves"]:
            old.append(edge.length)
            edge.length = edge.length * f
            out.append(lik.lnL())
        for (edge, _), length in zip(reversed(state["moves"]), reversed(old)):
            edge.length = length
            out.append(lik.lnL())
        return np.array(out)
    if kind == "sites":
        lik, out = state["lik"], []
        for what, value in state["proposals"]:
            _propose(lik, what, value)
            out.append(np.array(lik.siteLnLs()))
        _back(state)
        return out
    if kind == "batch":
        return state["batch"].run()
    if kind == "serve":
        server = state["server"]
        tickets = [server.submit(r) for r in state["requests"]]
        return np.array([server.wait(t)[0] for t in tickets])
    if kind == "mc3":
        m = state["mc3"]
        m.run(state["gens"])
        chains = [m.chain_state(i) for i in range(state["chains"])]
        return {k: np.stack([np.asarray(c[k]) for c in chains])
                for k in ("lnL", "heat", "parent", "len", "rates", "alpha")}
    rows, freqs, masks = compact(state["alignment"])
    return [rows, freqs, masks]


# -- what a pass cannot do without ----------------------------------------------

def _full(taxa, sites, kact, precision):
    """One full evaluation: every internal CL and its scaler written, the
    leaf masks and weights read (about 0.7 patterns a site; a rooted binary
    tree as the library sees it has taxa - 1 node updates at a leaf root).
    Multiply-adds: two 4x4 products and their product per component."""
    pat = 0.7 * sites
    row = 4 * kact * (4 if precision == "fp32" else 8) + (4 if precision == "fp32" else 8)
    leafy = 4 * kact * 8 * taxa * pat              # products with a leaf are lookups
    return {"bytes": pat * ((taxa - 1) * row + taxa + 12),
            "flops": max(pat * (taxa - 1) * kact * (2 * 28 + 4) - leafy, pat * kact * 8)}


def work(case):
    kind = case["kind"]
    kact = case.get("models", 1) * (case.get("ncat", 4) + (1 if case.get("pinv") else 0))
    if kind in ("proposals", "sites"):
        w = _full(case["taxa"], case["sites"], kact, case["precision"])
        return {k: v * case["n"] for k, v in w.items()}
    if kind == "branches":
        # About 1.5 log2(taxa) nodes on a path, each with a clean sibling.
        w = _full(case["taxa"], case["sites"], kact, case["precision"])
        part = 2 * case["n"] * 1.5 * math.log2(case["taxa"]) / case["taxa"]
        return {"bytes": 2 * w["bytes"] * part, "flops": w["flops"] * part}
    if kind in ("batch", "serve"):
        n = case["jobs"] if kind == "batch" else case["datasets"]
        each = 1.0 if kind == "batch" else case["requests"] / n
        ws = [_full(*_spread(case, j, n), kact, case["precision"]) for j in range(n)]
        return {k: each * sum(w[k] for w in ws) for k in ws[0]}
    if kind == "mc3":
        # A third of the moves are model moves (a full evaluation), the others
        # recompute a path.
        w = _full(case["taxa"], case["sites"], kact, case["precision"])
        part = min(1.0, 2 * 1.5 * math.log2(case["taxa"]) / case["taxa"])
        model = sum(v for k, v in _moves(case).items() if k in ("rates", "alpha")) / \
            sum(_moves(case).values())
        n = case["gens"] * case["chains"] * (model + (1 - model) * part)
        return {k: v * n for k, v in w.items()}
    cells = case["taxa"] * case["sites"]
    return {"bytes": cells * (1 + 2 * 0.6) + 4 * 2 * case["sites"],
            "flops": case["sites"] * math.log2(case["sites"])}


# -- the same results in plain 64-bit arithmetic ----------------------------------

def rate_matrix(m):
    pi = np.array(m["freqs"]) / np.sum(m["freqs"])
    R = np.zeros((4, 4))
    R[np.triu_indices(4, 1)] = m["rates"]
    R = R + R.T
    Q = R * pi[None, :]
    np.fill_diagonal(Q, 0.0)
    np.fill_diagonal(Q, -Q.sum(1))
    return Q


def eigen(m):
    """Q = V diag(lam) W of a reversible model, and its frequencies."""
    pi = np.array(m["freqs"]) / np.sum(m["freqs"])
    s = np.sqrt(pi)
    S = s[:, None] * rate_matrix(m) / s[None, :]
    lam, U = np.linalg.eigh(0.5 * (S + S.T))
    return lam, U / s[:, None], U.T * s[None, :], pi


def gamma_means(alpha, ncat):
    """Means of ncat equal-probability categories of a Gamma(alpha, 1/alpha)."""
    p = torch.arange(1, ncat, dtype=torch.float64) / ncat
    a = torch.full_like(p, alpha)
    lo, hi = torch.full_like(p, -700.0), torch.full_like(p, 7.0)   # ln of the cut
    for _ in range(200):
        mid = 0.5 * (lo + hi)
        below = torch.special.gammainc(a, mid.exp()) < p
        lo, hi = torch.where(below, mid, lo), torch.where(below, hi, mid)
    cuts = torch.special.gammainc(a + 1.0, (0.5 * (lo + hi)).exp())
    edges = [0.0] + [float(x) for x in cuts] + [1.0]
    return [ncat * (edges[i + 1] - edges[i]) for i in range(ncat)]


def _site_lnls(d, states, length, models, alpha):
    """ln likelihood of every column of `states` [taxa][n] (a device tensor)."""
    comps = []                                   # (model, weight, category rate)
    wsum = sum(d.weights)
    cats = gamma_means(alpha, d.ncat) if alpha is not None else [1.0]
    for i, w in enumerate(d.weights):
        comps += [(i, w / wsum * (1.0 - d.pinv) / len(cats), r) for r in cats]
        if d.pinv > 0.0:
            comps.append((i, w / wsum * d.pinv, 0.0))
    eig = [eigen(m) for m in models]
    qnorm = []                                   # mean rate of each raw Q
    for m, e in zip(models, eig):
        qnorm.append(float(-(e[3] * rate_matrix(m).diagonal()).sum()))
    mean = sum(w * qnorm[i] for i, w, r in comps if r != 0.0)
    P = np.zeros((len(d.kids), len(comps), 4, 4))
    for k, (i, w, r) in enumerate(comps):
        lam, V, W, _ = eig[i]
        P[:, k] = (V * np.exp(lam * (length * r / mean)[:, None, None])) @ W
    P = torch.tensor(np.maximum(P, 0.0), device=states.device)
    # Rows of a leaf: the state's indicator, all ones for a gap.
    table = torch.cat([torch.eye(4, dtype=torch.float64),
                       torch.ones(1, 4, dtype=torch.float64)]).to(states.device)
    cl, exps = {}, torch.zeros(states.shape[1], dtype=torch.float64, device=states.device)
    for v in reversed(d.order()):
        if not d.kids[v]:
            msg = (table @ P[v].transpose(1, 2))[:, states[d.leaf[v]].long()]
        else:
            a, b = d.kids[v]
            x = cl.pop(a) * cl.pop(b)            # [comps, n, 4]
            e = torch.frexp(x.amax((0, 2)))[1].to(torch.float64)
            exps += e
            x *= torch.exp2(-e)[None, :, None]
            if v == 0:
                break
            msg = x @ P[v].transpose(1, 2)
        cl[v] = msg
    like = torch.zeros_like(exps)
    for k, (i, w, _) in enumerate(comps):
        like += w * (x[k] @ torch.tensor(eig[i][3], device=x.device))
    return like.log() + exps * math.log(2.0)


def _columns(states):
    """Distinct columns, with counts: no need to prune a column twice."""
    cols, counts = np.unique(np.ascontiguousarray(states.T).view(
        np.dtype((np.void, states.shape[0]))).ravel(), return_counts=True)
    cols = cols.view(np.uint8).reshape(len(counts), -1)
    return torch.tensor(np.ascontiguousarray(cols.T), device="cuda"), counts


def _total(lnl, counts):
    return math.fsum((lnl.cpu().numpy() * counts).tolist())


def exact(case, seed):
    kind = case["kind"]
    if kind in ("mc3", "compact"):
        return None          # random walks, and whole numbers
    if kind == "batch":
        out = []
        for d in _jobs(case, seed):
            st, counts = _columns(d.states())
            out.append(_total(_site_lnls(d, st, d.len, d.models, d.alpha), counts))
        return np.array(out)
    if kind == "serve":
        sets, reqs = _requests(case, seed)
        cols = [_columns(d.states()) for d in sets]
        return np.array([_total(_site_lnls(r, cols[j][0], r.len, r.models, r.alpha), cols[j][1])
                         for j, r in reqs])
    d, rng = _data(case, seed)
    if kind == "branches":
        st, counts = _columns(d.states())
        node = {i: v for v, i in d.leaf.items()}
        length, out, trail = d.len.copy(), [], []
        # Branches of the root's two children are one branch of the unrooted
        # tree, so a leaf there rescales their sum.
        for i, f in _branches(d, rng, case["n"]):
            trail.append(length.copy())
            v = node[i]
            if d.up[v] == 0:
                for c in d.kids[0]:
                    length[c] *= f
            else:
                length[v] *= f
            out.append(_total(_site_lnls(d, st, length, d.models, d.alpha), counts))
        for length in reversed(trail):
            out.append(_total(_site_lnls(d, st, length, d.models, d.alpha), counts))
        return np.array(out)
    models, alpha = [dict(m) for m in d.models], d.alpha
    proposals = _proposals(d, rng, case["n"])
    if kind == "sites":
        st, counts = torch.tensor(d.states(), device="cuda"), 1
    else:
        st, counts = _columns(d.states())
    out = []
    for what, value in proposals:
        if what == "alpha":
            alpha = value
        else:
            models[0]["rates"] = value
        lnl = _site_lnls(d, st, d.len, models, alpha)
        out.append(lnl.cpu().numpy() * counts if kind == "sites" else _total(lnl, counts))
    return out if kind == "sites" else np.array(out)
