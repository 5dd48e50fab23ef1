"""Work that users of this library have it do, as cases whose time can be measured.

A case is a plain dict: the parameter set (tree and codon models), the task, the engine's
precision, the number of regions and the range of their lengths.  Region lengths follow from
the case alone (geometrically spaced over the range, in a mixed order); the alignment columns
are simulated from the seed, half from the coding and half from the noncoding model, with the
gaps and missing species of the benchmark's workloads.  Regions are handed over either as host
buffers in one call (``resident`` false: the command-line driver's path) or as a batch that is
already on the device (``resident`` true).
"""
import math
import random

import numpy as np
import torch

import phylocsf_gb300 as P
from phylocsf_gb300 import synth

# evaluations of one maximum-likelihood fit that no search can do without here: the two ends
# and the middle of the interval, the bracket's golden section point, about seven Brent steps
# to a 1 % bracket, and the returned value
EVALS_PER_FIT = 12
# evaluations of one OmegaModel score: two hypotheses x three rounds x two one-dimensional fits
EVALS_OMEGA = 12 * EVALS_PER_FIT


def _case(name, task, params, precision, regions, lo, hi, resident=True, strategy="mle"):
    return dict(name=name, task=task, params=params, precision=precision, regions=regions, lo=lo, hi=hi,
                resident=resident, strategy=strategy)


def listed():
    return [
        # one alignment scored at the default tree scale, as the command line does it (the
        # smallest call: launches and latency)
        _case("fly_one_fixed", "score", "12flies", "tf32x3b", 1, 300, 300, resident=False, strategy="fixed"),
        # one exon scored with the default maximum-likelihood strategy
        _case("mammal_one_mle", "score", "58mammals", "tf32x3b", 1, 137, 137, resident=False),
        # candidate regions of one transcript, all frames and sizes, short and ragged
        _case("mammal_orfs_mle", "score", "29mammals", "tf32x3b", 48, 25, 401, resident=False),
        # the headline workload's shape: exons and ORFs of 50-3,000 codons
        _case("mammal_batch_mle", "score", "58mammals", "tf32x3b", 384, 50, 3000),
        # whole genes on the vertebrate tree, where most columns are in long regions
        _case("vertebrate_genes_mle", "score", "100vertebrates", "tf32x3b", 60, 30, 10000),
        # many alignments at a fixed tree scale on the largest tree
        _case("mammal120_fixed", "score", "120mammals", "tf32x3b", 160, 100, 5000, strategy="fixed"),
        # log-likelihoods at given tree scales, every region with its own
        _case("mammal_lpr", "lpr", "58mammals", "fp32b", 301, 30, 2000),
        # the same in double precision, as a reference run
        _case("mammal_lpr_fp64", "lpr", "29mammals", "fp64", 24, 30, 900),
        # gradients with respect to every branch length and the tree scale (fitting a tree)
        _case("mammal_grad", "grad", "58mammals", "fp32b", 96, 50, 3000),
        # gradients of the parametric codon model (kappa, omega, rho, every branch)
        _case("vertebrate_omega_grad", "omega_grad", "100vertebrates", "fp32b", 40, 200, 2000),
        # the omega test of a few alignments
        _case("fly_omega_score", "omega_score", "12flies", "fp64", 6, 60, 400),
        # expected substitution counts of every branch (the E step of a rate fit)
        _case("mammal_counts", "counts", "29mammals", "fp32b", 64, 50, 1500),
    ]


def draw(rng: random.Random):
    """One more case of the same ranges, no larger than the largest listed one of its task."""

    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    task = rng.choice(["score_fixed", "score_mle", "score_mle", "lpr", "grad", "omega_grad", "omega_score", "counts"])
    if task == "score_fixed":
        c = _case("", "score", rng.choice(["12flies", "58mammals", "120mammals"]), "tf32x3b", spread(1, 160), 25, 5000,
                  resident=rng.random() < 0.5, strategy="fixed")
    elif task == "score_mle":
        params, most, longest = rng.choice([("12flies", 300, 3000), ("29mammals", 300, 3000), ("58mammals", 384, 3000),
                                            ("100vertebrates", 60, 10000)])
        c = _case("", "score", params, "tf32x3b", spread(1, most), 25, longest, resident=rng.random() < 0.5)
    elif task == "lpr":
        params, precision, most = rng.choice([("58mammals", "fp32b", 301), ("100vertebrates", "fp32b", 150),
                                              ("29mammals", "fp64", 24)])
        c = _case("", "lpr", params, precision, spread(1, most), 25, 900 if precision == "fp64" else 2000)
    elif task == "grad":
        c = _case("", "grad", rng.choice(["29mammals", "58mammals"]), "fp32b", spread(1, 96), 25, 3000)
    elif task == "omega_grad":
        c = _case("", "omega_grad", rng.choice(["12flies", "100vertebrates"]), "fp32b", spread(1, 40), 60, 2000)
    elif task == "omega_score":
        c = _case("", "omega_score", "12flies", "fp64", spread(1, 6), 60, 400)
    else:
        c = _case("", "counts", rng.choice(["12flies", "29mammals"]), "fp32b", spread(1, 64), 25, 1500)
    del c["name"]
    c["lo"] = spread(c["lo"], 4 * c["lo"])
    c["hi"] = max(c["lo"], spread(c["hi"] // 4, c["hi"]))
    return c


def _lengths(case):
    """Region lengths in codons: geometrically spaced from lo to hi, in a mixed order."""
    n = case["regions"]
    k = np.arange(n)
    f = k / (n - 1) if n > 1 else np.full(1, 0.5)
    L = np.rint(case["lo"] * (case["hi"] / case["lo"]) ** f).astype(np.int64)
    step = next(s for s in range(max(1, int(0.618 * n)), n + 2) if math.gcd(s, n) == 1)
    return L[(k * step) % n]


def _data(case, seed):
    """Simulated alignment columns: (parameter set, column offsets, leaf codes, random generator)."""
    ps = synth.load_params(case["params"])
    rng = np.random.default_rng(seed)
    n = case["regions"]
    gaps = synth.gap_fractions(rng, n, ps.tree.nl, 0.05, 0.40, 0.20)
    models = (np.arange(n) + int(rng.integers(0, 2))) % 2
    offs, leaves = synth.simulate(ps, _lengths(case), models.astype(np.int32), gaps, seed)
    return ps, offs, leaves, rng


def _points(case, rng):
    """Where lpr, gradients and counts are taken: one tree scale per region (and, for the
    parametric codon model, kappa and omega)."""
    n = case["regions"]
    rho = np.exp(rng.uniform(math.log(0.3), math.log(3.0), size=n))
    return rho, rng.uniform(1.5, 4.0, size=n), np.exp(rng.uniform(math.log(0.05), math.log(1.5), size=n))


def prepare(case, seed):
    ps, offs, leaves, rng = _data(case, seed)
    rho, kappa, omega = _points(case, rng)
    if case["task"].startswith("omega"):
        eng = P.Engine.for_tree(ps.tree, precision=case["precision"])
    else:
        eng = P.Engine(ps.tree, ps.S_c, ps.pi_c, ps.S_n, ps.pi_n, precision=case["precision"])
    state = dict(case=case, eng=eng, offs=offs, leaves=leaves, rho=rho, kappa=kappa, omega=omega)
    if case["resident"]:
        state["batch"] = eng.batch(offs, leaves)
    return state


def _fields(r):
    return {k: np.ascontiguousarray(r[k]) for k in r.dtype.names}


def run(state):
    case, eng = state["case"], state["eng"]
    task = case["task"]
    if task == "score":
        strategy = P.MLE if case["strategy"] == "mle" else P.FIXED
        if case["resident"]:
            return _fields(eng.score(state["batch"], strategy))
        return _fields(eng.score_batch(state["offs"], state["leaves"], strategy))
    if task == "omega_score":
        return _fields(eng.omega_score(state["batch"]))
    if task == "omega_grad":
        return eng.omega_grad(state["batch"], state["kappa"], state["omega"], state["rho"])
    if task == "lpr":
        return dict(zip(("lpr", "elpr", "status"), eng.lpr(state["batch"], 0, state["rho"])))
    if task == "grad":
        return dict(zip(("lpr", "d_branch", "d_rho", "status"), eng.grad(state["batch"], 0, state["rho"])))
    return dict(zip(("counts", "lpr", "status"), eng.branch_counts(state["batch"], 0, state["rho"])))


def work(case):
    nl = synth.load_params(case["params"]).tree.nl
    n, cols, nbr = case["regions"], int(_lengths(case).sum()), 2 * nl - 2
    inside = 8192.0 * (nl - 2) + 64.0 * (nl - 1) + 128.0   # one column, one evaluation
    p_set = 2.0 * 64 ** 3 * nbr                            # the P(t) of every branch
    outs, evals, p_sets = 10.0 * 8 * n, 1.0, float(n)
    per_col = inside
    if case["task"] == "score":
        evals = 2.0 * (EVALS_PER_FIT if case["strategy"] == "mle" else 1)
        p_sets = evals * n if case["strategy"] == "mle" else 2.0
    elif case["task"] == "omega_score":
        evals, p_sets = float(EVALS_OMEGA), float(EVALS_OMEGA * n)
    elif case["task"] == "grad":
        # outside products of the internal branches, and Q^T inter of every branch
        per_col, outs = inside + 8192.0 * (nl - 2) + 8192.0 * nbr, 8.0 * n * (nbr + 3)
    elif case["task"] == "omega_grad":
        # and two derivative forms of every branch
        per_col, outs = inside + 8192.0 * (nl - 2) + 3 * 8192.0 * nbr, 8.0 * n * (nbr + 5)
    elif case["task"] == "counts":
        # outside products, and a rank-one term of every branch's 64 x 64 counts
        per_col, outs = inside + 8192.0 * (nl - 2) + 8192.0 * nbr, 8.0 * n * nbr * 4096
    return {"bytes": float(cols * nl) + outs, "flops": evals * cols * per_col + p_sets * p_set}


# ---------------------------------------------------------------------------
# The same results in 64 bits with torch.

DEV = "cuda" if torch.cuda.is_available() else "cpu"
GOLDEN = 0.3819660
SQRT_EPS = 1.4901161193847656e-08


def _f64(x):
    return torch.as_tensor(np.asarray(x), dtype=torch.float64, device=DEV)


def _eigensystem(Q, pi):
    """(U, lambda, sqrt pi) of reversible rate matrices Q [..., 64, 64] with equilibrium pi."""
    sq = pi.sqrt()
    A = sq[..., :, None] * Q / sq[..., None, :]
    lam, U = torch.linalg.eigh(0.5 * (A + A.transpose(-1, -2)))
    return U, lam, sq


def _p_matrices(U, lam, sq, t):
    """P(t) = exp(tQ) [B, branches, 64, 64] for t [B, branches] and eigensystems [B, ...];
    negative off-diagonal entries are clamped and the diagonal makes each row sum to 1."""
    e = torch.expm1(lam[:, None, :] * t[:, :, None])
    E = torch.matmul(U[:, None] * e[:, :, None, :], U[:, None].transpose(-1, -2))
    E = E * sq[:, None, None, :] / sq[:, None, :, None]
    eye = torch.eye(64, dtype=torch.bool, device=E.device)
    E = E.clamp(min=0.0).masked_fill(eye, 0.0)
    return E + torch.diag_embed(1.0 - E.sum(-1))


def _inside(tree, Pm, prior, codes, ncols):
    """Per region of a group: (sum over its columns of log z, of the prior's expected log).
    Pm [B, branches, 64, 64], prior [B, 64], codes [B, L, leaves] (64 = any state)."""
    B, L, nl = codes.shape
    val = {}
    logs = torch.zeros((B, L), dtype=torch.float64, device=Pm.device)

    def partial(c):
        if c < nl:
            idx = codes[:, None, :, c].expand(B, 64, L)
            return torch.gather(torch.cat([Pm[:, c], Pm[:, c].sum(2, keepdim=True)], 2), 2, idx)
        return torch.matmul(Pm[:, c], val.pop(c))

    for node in range(nl, tree.n):
        l, r = [int(c) for c in np.flatnonzero(tree.parent == node)]
        v = partial(l) * partial(r)
        m = v.detach().amax(1).clamp(min=1e-300)
        val[node] = v / m[:, None]
        logs = logs + m.log()
    a = val[tree.n - 1]
    z = torch.einsum("bs,bsl->bl", prior, a)
    w = torch.einsum("bs,bsl->bl", prior * prior.log(), a) / z
    live = torch.arange(L, device=Pm.device)[None] < ncols[:, None]
    zero = torch.zeros((), dtype=torch.float64, device=Pm.device)
    return torch.where(live, z.log() + logs, zero).sum(1), torch.where(live, w, zero).sum(1)


class _Regions:
    """The regions of a case, evaluated in groups of similar length."""

    def __init__(self, tree, offs, leaves):
        self.tree, self.offs = tree, offs
        self.codes = torch.as_tensor(leaves, dtype=torch.uint8, device=DEV)
        self.branch = _f64(tree.branch[: tree.n - 1])
        self.len = np.diff(offs)

    def groups(self, regions):
        """Positions in `regions`, grouped so that little is spent on padding."""
        order = sorted(range(len(regions)), key=lambda k: -self.len[regions[k]])
        while order:
            longest = max(1, int(self.len[regions[order[0]]]))
            take = max(1, min(len(order), 60000 // longest, 64))
            take = max(1, sum(self.len[regions[k]] >= 0.7 * longest for k in order[:take]))
            yield order[:take]
            order = order[take:]

    def padded(self, regions):
        L = max(1, max(int(self.len[r]) for r in regions))
        out = torch.full((len(regions), L, self.tree.nl), 64, dtype=torch.int64, device=DEV)
        for k, r in enumerate(regions):
            out[k, : self.len[r]] = self.codes[self.offs[r]: self.offs[r + 1]].long()
        return out, torch.as_tensor([int(self.len[r]) for r in regions], device=DEV)

    def lpr(self, regions, model, rho, systems, priors):
        """lpr and elpr of requests: regions, rows of `systems` and `priors`, tree scales."""
        lp, el = np.zeros(len(regions)), np.zeros(len(regions))
        for g in self.groups(regions):
            m = torch.as_tensor([model[k] for k in g], device=DEV)
            t = _f64([rho[k] for k in g])[:, None] * self.branch[None]
            codes, n = self.padded([regions[k] for k in g])
            a, b = _inside(self.tree, _p_matrices(*[x[m] for x in systems], t), priors[m], codes, n)
            lp[g], el[g] = a.cpu().numpy(), b.cpu().numpy()
        return lp, el


def _uniforms():
    """The deterministic stream of restart points (SplitMix64 from 0)."""
    s, mask = 0, (1 << 64) - 1
    while True:
        s = (s + 0x9E3779B97F4A7C15) & mask
        z = s
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        yield ((z ^ (z >> 31)) >> 11) / 9007199254740992.0


def _fit(lo, hi, init, accuracy=0.01):
    """Maximise over [lo, hi]: yields points, is sent their values, returns (point, value)."""
    flo, fhi = (yield lo), (yield hi)
    x, fx, u = init, (yield init), _uniforms()
    for tries in range(251):
        if not (fx <= flo or fx <= fhi):
            break
        if tries == 250:
            x = lo if flo > fhi else hi
            break
        x = math.exp(math.log(lo) + next(u) * (math.log(hi) - math.log(lo)))
        fx = yield x
    if not lo < x < hi:
        return x, (yield x)
    a, b, z, fz = lo, hi, x, -fx                       # Brent's method on -f
    v = w = a + GOLDEN * (b - a)
    fv = fw = -(yield v)
    d = e = 0.0
    for _ in range(1000):
        mid, tol = 0.5 * (a + b), SQRT_EPS * abs(z)
        p = q = r = 0.0
        step, last = e, d
        if abs(last) > tol:
            r, q = (z - w) * (fz - fv), (z - v) * (fz - fw)
            p, q = (z - v) * q - (z - w) * r, 2.0 * (q - r)
            p, q = (-p, q) if q > 0.0 else (p, -q)
            r, last = last, step
        if abs(p) < abs(0.5 * q * r) and p < q * (z - a) and p < q * (b - z):
            step = p / q
            if (z + step - a) < 2.0 * tol or (b - z - step) < 2.0 * tol:
                step = tol if z < mid else -tol
        else:
            last = (b - z) if z < mid else -(z - a)
            step = GOLDEN * last
        e, d = last, step
        n = z + (step if abs(step) >= tol else (tol if step > 0.0 else -tol))
        fn = -(yield n)
        if fn <= fz:
            a, b = (a, z) if n < z else (z, b)
            v, fv, w, fw, z, fz = w, fw, z, fz, n, fn
        else:
            a, b = (n, b) if n < z else (a, n)
            if fn <= fw or w == z:
                v, fv, w, fw = w, fw, n, fn
            elif fn <= fv or v == z or v == w:
                v, fv = n, fn
        if not (b - a) / z > accuracy:
            break
    return z, -fz


def _lockstep(fits, evaluate):
    """Advance generators together: evaluate([(key, point)]) -> values, until all returned."""
    out, ask = {}, {}
    for k, f in fits.items():
        ask[k] = next(f)
    while ask:
        keys = list(ask)
        val = evaluate([(k, ask[k]) for k in keys])
        for k, y in zip(keys, val):
            try:
                ask[k] = fits[k].send(float(y))
            except StopIteration as stop:
                out[k] = stop.value
                del ask[k]
    return out


def _rate_matrix(S, pi):
    """q_ij = s_ij pi_j with zero row sums and a mean rate of 1."""
    Q = S * pi[None, :]
    np.fill_diagonal(Q, 0.0)
    np.fill_diagonal(Q, -Q.sum(1))
    return Q / (-(pi * np.diag(Q)).sum())


def _fixed_models(ps):
    Q = _f64(np.stack([_rate_matrix(ps.S_c, ps.pi_c), _rate_matrix(ps.S_n, ps.pi_n)]))
    pi = _f64(np.stack([ps.pi_c, ps.pi_n]))
    return Q, pi


_AA = "KNKNTTTTRSRSIIMIQHQHPPPPRRRRLLLLEDEDAAAAGGGGVVVV*Y*YSSSS*CWCLFLF"
_STOPS = [48, 50, 56]


def _omega_q(f3x4, kappa, omega, sigma):
    """(Q, pi) of the parametric codon model; kappa and omega may carry gradients."""
    nuc = torch.as_tensor([[i // 16, (i // 4) % 4, i % 4] for i in range(64)], device=DEV)
    rel = torch.ones((3, 4), dtype=torch.float64, device=DEV)
    rel[:, :3] = f3x4.reshape(3, 3)
    pos = rel / rel.sum(1, keepdim=True)
    sc = pos[0][nuc[:, 0]] * pos[1][nuc[:, 1]] * pos[2][nuc[:, 2]]
    pi = sc / (1.0 - (1.0 - sigma) * sc[_STOPS].sum())
    diff = nuc[:, None] != nuc[None]
    one = diff.sum(2) == 1
    a = torch.where(diff, nuc[:, None], -1).amax(2)
    b = torch.where(diff, nuc[None], -1).amax(2)
    lo, hi = torch.minimum(a, b), torch.maximum(a, b)
    transition = one & (((lo == 0) & (hi == 2)) | ((lo == 1) & (hi == 3)))
    aa = torch.as_tensor([ord(c) for c in _AA], device=DEV)
    stop = torch.zeros(64, dtype=torch.bool, device=DEV)
    stop[_STOPS] = True
    nonsyn = one & ~stop[:, None] & ~stop[None] & (aa[:, None] != aa[None])
    zero = torch.zeros((), dtype=torch.float64, device=DEV)
    R = torch.where(one, pi[None, :], zero) * torch.where(transition, kappa, zero + 1) * torch.where(nonsyn, omega, zero + 1)
    R = R - torch.diag(R.sum(1))
    return R / -(pi * R.diagonal()).sum(), pi


def _f3x4(codes):
    """Nucleotide counts (pseudocount 1) per codon position relative to T."""
    c = codes[codes < 64].astype(np.int64)
    n = np.stack([np.bincount((c >> s) & 3, minlength=4) + 1.0 for s in (4, 2, 0)])
    return (n[:, :3] / n[:, 3:]).reshape(-1)


def _exact_score(case, ps, offs, leaves):
    reg = _Regions(ps.tree, offs, leaves)
    Q, pi = _fixed_models(ps)
    systems = _eigensystem(Q, pi)
    n = case["regions"]
    fits = [(r, m) for r in range(n) for m in (0, 1)]
    rho = dict.fromkeys(fits, 1.0)
    if case["strategy"] == "mle":
        def evaluate(asked):
            return reg.lpr([k[0] for k, _ in asked], [k[1] for k, _ in asked], [x for _, x in asked], systems, pi)[0]

        rho = {k: v[0] for k, v in _lockstep({k: _fit(1e-2, 10.0, 1.0) for k in fits}, evaluate).items()}
    rhos = np.array([rho[k] for k in fits])
    lpr, elpr = reg.lpr([k[0] for k in fits], [k[1] for k in fits], rhos, systems, pi)
    db = 10.0 / math.log(10.0)
    return {"score": db * (lpr[0::2] - lpr[1::2]), "anc_comp_score": db * (elpr[0::2] - elpr[1::2]),
            "rho_c": rhos[0::2], "rho_n": rhos[1::2], "lpr_c": lpr[0::2], "lpr_n": lpr[1::2],
            "elpr_c": elpr[0::2], "elpr_n": elpr[1::2], "status": np.zeros(n, np.int32), "evals": None}


def _exact_adjoint(case, ps, offs, leaves, rho):
    """Region by region: lpr, d lpr / d P and P, for gradients and expected counts."""
    reg = _Regions(ps.tree, offs, leaves)
    Q, pi = _fixed_models(ps)
    systems = [x[:1] for x in _eigensystem(Q, pi)]
    lpr, grads, counts = [], [], []
    for r in range(case["regions"]):
        Pm = _p_matrices(*systems, rho[r] * reg.branch[None]).requires_grad_(True)
        codes, n = reg.padded([r])
        lp, _ = _inside(ps.tree, Pm, pi[:1], codes, n)
        lp.sum().backward()
        lpr.append(float(lp.detach()))
        if case["task"] == "grad":
            grads.append((Pm.grad * torch.matmul(Q[0], Pm.detach())).sum((2, 3))[0].cpu().numpy())
        else:
            counts.append((Pm.grad * Pm.detach())[0].cpu().numpy())
    status = np.zeros(case["regions"], np.int32)
    if case["task"] == "grad":
        d = np.stack(grads)
        return {"lpr": np.array(lpr), "d_branch": d, "d_rho": d @ ps.tree.branch[: ps.tree.n - 1], "status": status}
    return {"counts": np.stack(counts), "lpr": np.array(lpr), "status": status}


def _exact_omega_grad(case, ps, offs, leaves, rho, kappa, omega):
    reg = _Regions(ps.tree, offs, leaves)
    out = {k: [] for k in ("lpr", "d_branch", "d_rho", "d_kappa", "d_omega")}
    for r in range(case["regions"]):
        x = _f64([kappa[r], omega[r]]).requires_grad_(True)
        Q, pi = _omega_q(_f64(_f3x4(leaves[offs[r]: offs[r + 1]])), x[0], x[1], 1.0)
        t = (rho[r] * reg.branch).requires_grad_(True)
        # exp(tQ), branch by branch in blocks (its derivative in Q and t comes from autograd)
        Pm = torch.cat([torch.linalg.matrix_exp(t[k: k + 32, None, None] * Q) for k in range(0, len(t), 32)])
        Pl = Pm.detach()[None].requires_grad_(True)
        codes, n = reg.padded([r])
        lp, _ = _inside(ps.tree, Pl, (pi / pi.sum()).detach()[None], codes, n)
        lp.sum().backward()
        Pm.backward(Pl.grad[0])
        out["lpr"].append(float(lp.detach()))
        out["d_branch"].append(t.grad.cpu().numpy())
        out["d_rho"].append(float((t.grad * reg.branch).sum()))
        out["d_kappa"].append(float(x.grad[0]))
        out["d_omega"].append(float(x.grad[1]))
    return dict({k: np.array(v) for k, v in out.items()}, status=np.zeros(case["regions"], np.int32))


def _log_prior(kind, x):
    if kind == "rho":                                      # half-Cauchy, mode 1, scale 0.5
        density = 1.0 / (math.pi * 0.5 * (1.0 + ((x - 1.0) / 0.5) ** 2))
        return math.log(density) - math.log(1.0 - (math.atan(-1.0 / 0.5) / math.pi + 0.5))
    y = x - 1.0 + 2.220446049250313e-16                    # Gamma(7, 0.25) of kappa - 1
    return 6.0 * math.log(y) - y / 0.25 - math.lgamma(7.0) - 7.0 * math.log(0.25)


def _exact_omega_score(case, ps, offs, leaves, omega_h1=0.2, sigma_h1=0.01):
    reg = _Regions(ps.tree, offs, leaves)
    n = case["regions"]
    freq = [_f64(_f3x4(leaves[offs[r]: offs[r + 1]])) for r in range(n)]

    def region():
        """Coordinate ascent under both hypotheses; yields (omega, sigma, rho, kappa)."""
        rho, kappa, res = 1.0, 2.5, []
        for omega, sigma in ((1.0, 1.0), (omega_h1, sigma_h1)):
            for _ in range(3):
                for kind, lo, init in (("rho", 0.001, rho), ("kappa", 1.0, kappa)):
                    f = _fit(lo, 10.0, init)
                    x = next(f)
                    while True:
                        y = yield (omega, sigma) + ((x, kappa) if kind == "rho" else (rho, x))
                        try:
                            x = f.send(y + _log_prior(kind, x))
                        except StopIteration as stop:
                            best, value = stop.value
                            break
                    rho, kappa = (best, kappa) if kind == "rho" else (rho, best)
            res += [value, rho, kappa]
        return res

    def evaluate(asked):
        Qp = [_omega_q(freq[r], _f64(k), _f64(o), s) for r, (o, s, _, k) in asked]
        Q, pi = torch.stack([q for q, _ in Qp]), torch.stack([p for _, p in Qp])
        prior = pi / pi.sum(1, keepdim=True)
        return reg.lpr([r for r, _ in asked], list(range(len(asked))), [x[2] for _, x in asked], _eigensystem(Q, pi), prior)[0]

    res = _lockstep({r: region() for r in range(n)}, evaluate)
    l0, r0, k0, l1, r1, k1 = np.array([res[r] for r in range(n)]).T
    return {"score": 10.0 * (l1 - l0) / math.log(10.0), "lpr_h0": l0, "lpr_h1": l1, "rho_h0": r0, "kappa_h0": k0,
            "rho_h1": r1, "kappa_h1": k1, "status": np.zeros(n, np.int32), "evals": None}


def exact(case, seed):
    ps, offs, leaves, rng = _data(case, seed)
    rho, kappa, omega = _points(case, rng)
    if case["task"] == "score":
        return _exact_score(case, ps, offs, leaves)
    if case["task"] == "lpr":
        reg = _Regions(ps.tree, offs, leaves)
        Q, pi = _fixed_models(ps)
        n = case["regions"]
        lpr, elpr = reg.lpr(list(range(n)), [0] * n, rho, _eigensystem(Q, pi), pi)
        return {"lpr": lpr, "elpr": elpr, "status": np.zeros(n, np.int32)}
    if case["task"] == "omega_grad":
        return _exact_omega_grad(case, ps, offs, leaves, rho, kappa, omega)
    if case["task"] == "omega_score":
        return _exact_omega_score(case, ps, offs, leaves)
    return _exact_adjoint(case, ps, offs, leaves, rho)
