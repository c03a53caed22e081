"""What a user of subby_gb300 has it do: the timed cases.

A case is a tree, a substitution model and an alignment, and one of the
package's calls on them:

  run        Plan.run on device tensors (logLike, counts, rootProb)
  host       Plan.run on pinned host arrays (copies in and out are part of it)
  gamma      LogLike over K discrete-gamma rate categories (a ``*H`` model)
  posterior  Plan.posteriors, every node
  grad       Plan.grad: logLike with branch-length and exchangeability gradients

Alignments are simulated down the tree on the GPU: internal rows are
unobserved (token A), leaf cells carry the simulated state or, at the case's
rate, a gap (A + 1) or an unobserved cell (A).
"""
import math

import numpy as np
import torch

import subby_gb300 as sg
from subby_gb300 import models, synth


def _case(name, call, A, model, leaves, C, **more):
    c = {"name": name, "call": call, "A": A, "model": model, "leaves": leaves, "C": C, "branch": 0.08, "gap": 0.1,
         "unobserved": 0.02, "loglike": True, "counts": True, "rootprob": False, "f81": False, "masked": True}
    c.update(more)
    return c


def listed():
    return [
        # one short DNA block (a gene, an MAF block): launch latency counts
        _case("dna_small", "run", 4, "hky85", 16, 1024, rootprob=True, unobserved=0.025, gap=0.025, branch=0.1),
        # genome-scale DNA counts on a 128-species tree, the headline workload
        _case("dna_counts", "run", 4, "hky85", 128, 1 << 20, loglike=False, branch=0.05, unobserved=0.0),
        # counts over a large species tree (the largest of the serving stream)
        _case("dna_deep_counts", "run", 4, "hky85", 512, 50001, branch=0.1, gap=0.05),
        # rate heterogeneity: likelihoods of four gamma categories
        _case("dna_gamma_loglike", "gamma", 4, "hky85", 100, 200003, counts=False, categories=4, alpha=0.5),
        # the same counts called on host buffers
        _case("dna_host_counts", "host", 4, "f81", 64, 1 << 18, f81=True),
        # ancestral reconstruction: posteriors of every node
        _case("dna_posterior", "posterior", 4, "hky85", 64, 100001, counts=False),
        # paired RNA columns (16 states), one family of a few thousand pairs
        _case("rna16_counts", "run", 16, "reversible", 50, 4003, gap=0.05),
        # protein counts of a medium alignment
        _case("protein_counts", "run", 20, "reversible", 100, 20011),
        # training step of a protein model: likelihood and both gradients
        _case("protein_grad", "grad", 20, "reversible", 200, 100000, gap=0.15, unobserved=0.0),
        # a non-reversible protein model
        _case("irrev_counts", "run", 20, "irreversible", 50, 8001),
        # 64-state (codon-sized) counts with near-degenerate eigenvalues
        _case("codon_counts", "run", 64, "degenerate", 64, 65536, loglike=False, gap=0.0, unobserved=0.0, branch=0.1),
        # 64-state F81 fast path
        _case("codon_f81_counts", "run", 64, "f81", 64, 20011, f81=True, branch=0.1, gap=0.05),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same ranges: trees of 8 to 512 leaves, 100 to 2^20 columns."""
    kind = rng.choice(["small", "dna", "deep", "gamma", "host", "posterior", "rna16", "protein", "grad", "irrev",
                       "codon", "codon_f81"])
    more = {"gap": round(rng.uniform(0.0, 0.2), 3), "unobserved": round(rng.uniform(0.0, 0.03), 3),
            "branch": round(math.exp(rng.uniform(math.log(0.03), math.log(0.2))), 4),
            "loglike": rng.random() < 0.5, "masked": rng.random() < 0.75}
    dna = rng.choice(["hky85", "f81", "jc"])
    fast = dna != "hky85" and rng.random() < 0.5

    def make(call, A, model, leaves, C, most, **m):
        # the work of one pass stays under that of the largest listed case
        C = max(100, min(C, most // (2 * leaves - 1)))
        c = _case("", call, A, model, leaves, C, **dict(more, **m))
        del c["name"]
        return c

    if kind == "small":
        return make("run", 4, dna, _log(rng, 8, 64), _log(rng, 100, 20000), 255 << 20, rootprob=rng.random() < 0.5,
                    f81=fast)
    if kind == "dna":
        return make("run", 4, dna, _log(rng, 8, 128), _log(rng, 1 << 14, 1 << 20), 200 << 20, f81=fast)
    if kind == "deep":
        return make("run", 4, dna, _log(rng, 129, 512), _log(rng, 1000, 60000), 1023 * 50000, f81=fast)
    if kind == "gamma":
        return make("gamma", 4, dna, _log(rng, 8, 256), _log(rng, 1000, 400000), 100 << 20, counts=False,
                    categories=rng.choice([2, 4, 6]), alpha=round(rng.uniform(0.2, 2.0), 3))
    if kind == "host":
        return make("host", 4, dna, _log(rng, 8, 128), _log(rng, 1000, 1 << 18), 40 << 20, f81=fast)
    if kind == "posterior":
        return make("posterior", 4, dna, _log(rng, 8, 128), _log(rng, 1000, 200000), 20 << 20, counts=False)
    if kind == "rna16":
        return make("run", 16, "reversible", _log(rng, 8, 200), _log(rng, 200, 50000), 4 << 20)
    if kind == "protein":
        return make("run", 20, "reversible", _log(rng, 8, 400), _log(rng, 200, 50000), 10 << 20)
    if kind == "grad":
        return make("grad", 20, "reversible", _log(rng, 16, 256), _log(rng, 1000, 100000), 30 << 20)
    if kind == "irrev":
        A = rng.choice([4, 16, 20])
        return make("run", A, "irreversible", _log(rng, 8, 128), _log(rng, 200, 20000), (8 << 20) if A == 4 else 800000)
    f81 = kind == "codon_f81"
    return make("run", 64, "f81" if f81 else "reversible", _log(rng, 8, 200), _log(rng, 100, 65536), 7 << 20, f81=f81)


def _tree_model(case, seed):
    rng = np.random.default_rng([seed, case["A"], case["leaves"]])
    A = case["A"]
    pi = rng.dirichlet(np.full(A, 2.0))
    if case["model"] == "hky85":
        model = models.hky85_diag(2.0, pi)
    elif case["model"] == "jc":
        model = models.jukes_cantor_model(A)
    elif case["model"] == "f81":
        model = models.f81_model(pi)
    elif case["model"] == "irreversible":
        model = models.random_irreversible(A, rng)
    elif case["model"] == "degenerate":
        model = models.near_degenerate_reversible(A, rng, dirichlet_alpha=2.0)[0]
    else:
        model = models.random_reversible(A, rng, 0.5, 2.0)[0]
    return synth.random_tree(case["leaves"], case["branch"], rng), model


def _leaves(parent):
    leaf = np.ones(len(parent), dtype=bool)
    leaf[parent[1:]] = False
    return leaf


def _tokens(case, seed, tree, model):
    """(R, C) int32 tokens simulated down the tree, on the GPU."""
    A, C, parent = case["A"], case["C"], tree.parentIndex
    M = synth.sub_matrices64(model, tree.distanceToParent)
    cum = torch.as_tensor(np.cumsum(M, axis=-1)[..., :-1].astype(np.float32)).cuda().contiguous()
    g = torch.Generator(device="cuda").manual_seed(seed)
    top = torch.as_tensor(np.cumsum(np.asarray(model.pi))[:-1].astype(np.float32)).cuda()
    R = len(parent)
    out = torch.empty((R, C), dtype=torch.int32, device="cuda")
    out[0] = torch.searchsorted(top, torch.rand(C, generator=g, device="cuda"), right=True)
    for n in range(1, R):
        u = torch.rand(C, generator=g, device="cuda")
        out[n] = (u[:, None] >= cum[n][out[parent[n]].long()]).sum(1)
    leaf = _leaves(parent)
    for n in range(R):
        if not leaf[n]:
            out[n] = A
            continue
        u = torch.rand(C, generator=g, device="cuda")
        out[n] = torch.where(u < case["gap"], A + 1, torch.where(u < case["gap"] + case["unobserved"], A, out[n]))
    return out


def prepare(case, seed):
    tree, model = _tree_model(case, seed)
    aln = _tokens(case, seed, tree, model)
    state = {"case": case}
    call, A, C = case["call"], case["A"], case["C"]
    if call == "gamma":
        rates, _ = models.gamma_rate_categories(case["alpha"], case["categories"])
        state.update(aln=aln, tree=tree, model=models.scale_model(model, rates))
        sg.LogLike(aln[:, :1].contiguous(), tree, state["model"])  # the cached plans
        return state
    state["plan"] = sg.Plan(tree, model)
    if call == "host":
        pin = torch.empty(tuple(aln.shape), dtype=torch.int32, pin_memory=True)
        pin.copy_(aln)
        state["aln"] = pin.numpy()
        state["out"] = {"logLike": torch.empty(C, pin_memory=True).numpy(),
                        "counts": torch.empty((A, A, C), pin_memory=True).numpy()}
        state["kept"] = pin
    elif call == "grad":
        pin = torch.empty(tuple(aln.shape), dtype=torch.int32, pin_memory=True)
        pin.copy_(aln)
        state["aln"], state["kept"] = pin.numpy(), pin
        state["g"] = _cotangent(case, seed).astype(np.float32)
    else:
        state["aln"] = aln
    return state


def _cotangent(case, seed):
    # site weights (pattern multiplicities) of the training objective
    return np.random.default_rng([seed, 9]).integers(1, 5, size=case["C"]).astype(np.float64)


def run(state):
    case = state["case"]
    call = case["call"]
    if call == "gamma":
        return sg.LogLike(state["aln"], state["tree"], state["model"])
    plan = state["plan"]
    if call == "posterior":
        return plan.posteriors(state["aln"])["node"]
    if call == "grad":
        return plan.grad(state["aln"], state["g"])
    return plan.run(state["aln"], loglike=case["loglike"], counts=case["counts"], rootprob=case["rootprob"],
                    f81=case["f81"], branch_mask="auto" if case["masked"] else None, out=state.get("out"))


def work(case):
    A, C, L = case["A"], case["C"], case["leaves"]
    R, inner = 2 * L - 1, L - 2   # nodes; internal nodes below the root
    by, fl = 4.0 * R * C, 2.0 * A * A * inner * C
    call = case["call"]
    if call == "gamma":
        return {"bytes": by + 4.0 * C * case["categories"], "flops": fl * case["categories"]}
    if call == "posterior":
        return {"bytes": by + 4.0 * R * A * C, "flops": fl + (2.0 * A * A + 2 * A) * (R - 1) * C}
    outside = 2.0 * A * A * inner                    # D^T M
    if call == "grad":
        return {"bytes": by + 4.0 * C * 2 + 8.0 * (R + A * A),
                "flops": fl + (outside + 2.0 * A * A * (R - 1 + inner) + 2.0 * A * A * (R - 1)) * C}
    by += 4.0 * C * (A * A + (1 if case["loglike"] else 0) + (A if case["rootprob"] else 0))
    if case["f81"]:
        # closed-form products: O(A) a branch, the rank-one accumulation A^2
        return {"bytes": by, "flops": (2.0 * A * inner * 4 + 2.0 * A * A * (R - 1)) * C}
    if case["model"] == "irreversible":
        # complex projections, accumulation and back-transform
        per = outside + 4.0 * A * A * (R - 1 + inner) + 14.0 * A * A * (R - 1) + 12.0 * A ** 3
    else:
        per = outside + 2.0 * A * A * (R - 1 + inner) + 3.0 * A * A * (R - 1) + 4.0 * A ** 3
    return {"bytes": by, "flops": fl + per * C}


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch: per-column inside and outside passes
# with every node's vectors kept, the eigenbasis accumulation and its
# back-transform


def _mask(tok, parent, leaf, A):
    """Branches of the Steiner tree of a column's ungapped leaves."""
    R = len(parent)
    ung = [(tok[n] >= 0) & (tok[n] <= A) if leaf[n] else torch.zeros_like(tok[n], dtype=torch.bool) for n in range(R)]
    has, many = [u.clone() for u in ung], [torch.zeros_like(tok[0]) for _ in range(R)]
    for n in range(R - 1, 0, -1):
        has[parent[n]] |= has[n]
        many[parent[n]] += has[n]
    st = [ung[n] | (many[n] >= 2) for n in range(R)]
    for n in range(1, R):
        st[n] |= st[parent[n]] & has[n]
    return [st[n] & st[parent[n]] for n in range(1, R)]


def _scaled(x):
    m = x.max(0).values
    m = torch.where(m > 0, m, torch.ones_like(m))
    return x / m, torch.log(m)


class _Exact:
    def __init__(self, tree, model):
        self.parent = np.asarray(tree.parentIndex)
        self.leaf = _leaves(self.parent)
        t = np.asarray(tree.distanceToParent, np.float64)
        mu, V, pi = np.asarray(model.eigenvalues), np.asarray(model.eigenvectors), np.asarray(model.pi, np.float64)
        self.irrev = hasattr(model, "eigenvectors_inv")
        E = np.exp(mu[None, :] * t[:, None])
        if self.irrev:
            Vi = np.asarray(model.eigenvectors_inv)
            self.M = np.einsum("ik,rk,kj->rij", V, E, Vi).real
            # the reference's formula: D by V^-1, U by V, back by V C V^-1
            self.down, self.up, self.left, self.right = Vi, V.T, V, Vi
            self.rate = (V * mu) @ Vi
        else:
            sp = np.sqrt(pi)
            self.M = np.einsum("ik,rk,jk->rij", V, E, V) / sp[None, :, None] * sp[None, None, :]
            self.down, self.up, self.left, self.right = (V / sp[:, None]).T, (V * sp[:, None]).T, V, V.T
            self.rate = (V * mu) @ V.T
        d = mu[:, None] - mu[None, :]
        near = np.abs(d) < 1e-8
        J = (E[:, None, :] * np.expm1(d[None] * t[:, None, None])) / np.where(near, 1.0, d)[None]
        self.J = np.where(near[None], t[:, None, None] * E[:, :, None], J)
        self.dE = mu[None, :] * E
        for k in ("M", "down", "up", "left", "right", "rate", "J", "dE"):
            setattr(self, k, torch.as_tensor(np.ascontiguousarray(getattr(self, k))).cuda())
        self.pi = torch.as_tensor(pi).cuda()
        self.A, self.R = len(pi), len(self.parent)
        self.kids = [[] for _ in range(self.R)]
        for n in range(1, self.R):
            self.kids[self.parent[n]].append(n)

    def inside(self, tok):
        A, R = self.A, self.R
        row = torch.arange(A, device="cuda")[:, None]
        self.obs = lambda n: ((tok[n] == row) | (tok[n] < 0) | (tok[n] >= A)).double()
        self.U, self.CC, self.lnU = [None] * R, [None] * R, [0.0] * R
        for n in range(R - 1, -1, -1):
            u, ln = self.obs(n), 0.0
            for k in self.kids[n]:
                u, ln = u * self.CC[k], ln + self.lnU[k]
            u, e = _scaled(u)
            self.U[n], self.lnU[n] = u, ln + e
            if n:
                self.CC[n] = self.M[n] @ u
        p = self.pi @ self.U[0]
        self.lnL = torch.log(p) + self.lnU[0]
        return self.lnL

    def root(self):
        q = self.pi[:, None] * self.U[0]
        return q / q.sum(0)

    def outside(self):
        """(n, D_n scaled by the branch weight) of every branch, parents first."""
        O, lnO = {0: self.pi[:, None] * self.obs(0)}, {0: 0.0}
        for n in range(self.R):
            for k, sib in zip(self.kids[n], self.kids[n][::-1]):
                D, e = _scaled(O[n] * self.CC[sib])
                lnD = lnO[n] + self.lnU[sib] + e
                yield k, D * torch.exp(lnD + self.lnU[k] - self.lnL)
                if self.kids[k]:
                    O[k], lnO[k] = (self.M[k].T @ D) * self.obs(k), lnD
            O.pop(n, None), lnO.pop(n, None)

    def counts(self, tok, masked):
        A, c = self.A, tok.shape[1]
        acc = torch.zeros((A, A, c), dtype=self.J.dtype, device="cuda")
        mask = _mask(tok, self.parent, self.leaf, A) if masked else None
        for n, D in self.outside():
            if masked:
                D = D * mask[n - 1]
            acc += self.J[n][:, :, None] * (self.down @ D.to(self.J.dtype))[:, None] * (self.up @ self.U[n].to(
                self.J.dtype))[None]
        x = (self.left @ acc.reshape(A, A * c)).reshape(A, A, c)
        x = torch.matmul(self.right.T, x)
        diag = torch.eye(A, device="cuda", dtype=torch.bool)[:, :, None]
        x = torch.where(diag, x, x * self.rate[:, :, None])
        return x.real if self.irrev else x

    def grad(self, g):
        """Sums over the columns of g: (R,) branch lengths, (A, A) X_n * J_n in the eigenbasis."""
        dt = torch.zeros(self.R, dtype=torch.float64, device="cuda")
        X = torch.zeros((self.A, self.A), dtype=torch.float64, device="cuda")
        for n, D in self.outside():
            x = ((self.down @ D) * g) @ (self.up @ self.U[n]).T
            dt[n] = (self.dE[n] * x.diagonal()).sum()
            X += self.J[n] * x
        return dt, X

    def posteriors(self):
        out = torch.empty((self.R, self.A, self.lnL.shape[0]), dtype=torch.float64, device="cuda")
        out[0] = self.root()
        for n, D in self.outside():
            q = (self.M[n].T @ D) * self.U[n]
            out[n] = q / q.sum(0)
        return out


def exact(case, seed):
    tree, model = _tree_model(case, seed)
    tok = _tokens(case, seed, tree, model)
    A, C, R = case["A"], case["C"], tok.shape[0]
    step = max(256, int(6e9 / (8 * A * (3 * R + 8 * A))))
    call = case["call"]
    cuts = [tok[:, c:c + step].long() for c in range(0, C, step)]
    if call == "gamma":
        rates, _ = models.gamma_rate_categories(case["alpha"], case["categories"])
        rows = []
        for r in np.asarray(rates):
            x = _Exact(tree, models.scale_model(model, float(r)))
            rows.append(torch.cat([x.inside(t) for t in cuts]))
        return torch.stack(rows)
    x = _Exact(tree, model)
    if call == "posterior":
        parts = []
        for t in cuts:
            x.inside(t)
            parts.append(x.posteriors())
        return torch.cat(parts, -1)
    if call == "grad":
        g = torch.as_tensor(_cotangent(case, seed)).cuda()
        ll, dt, X = [], 0.0, 0.0
        for i, t in enumerate(cuts):
            ll.append(x.inside(t))
            a, b = x.grad(g[i * step:i * step + t.shape[1]])
            dt, X = dt + a, X + b
        return torch.cat(ll), dt, x.left @ X @ x.right
    got = {"logLike": [], "counts": [], "rootProb": []}
    for t in cuts:
        got["logLike"].append(x.inside(t))
        if case["rootprob"]:
            got["rootProb"].append(x.root())
        if case["counts"]:
            got["counts"].append(x.counts(t, case["masked"]))
    want = {"logLike": case["loglike"], "counts": case["counts"], "rootProb": case["rootprob"]}
    if call == "host":   # the caller's buffers: both are filled as asked
        want["rootProb"] = False
    return {k: torch.cat(v, -1) for k, v in got.items() if want[k] and v}
