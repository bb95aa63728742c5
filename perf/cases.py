"""Workloads of this package's public entry points, for timing and for checking.

Every case is one call sequence that a user's program makes, named by what it is:

  compute    TransferEntropyEngine(data, names[, sources]).compute(...) on a host
             expression matrix, to the host TE matrix (discretisation or
             binarisation, kernel choice and assembly included)
  matrix     raw integer bins already on the device -> dense relabelling,
             coarsening where the bins need it, all ordered pairs -> device matrix
  binary     the GEMM-B2 matrix of 0/1 bins already on the device
  surrogate  NetWeaver(result).infer("surrogate_test"): the block-shuffle test, full
             or with the learned null
  fdr        NetWeaver((matrix, names)).infer("fdr"): thresholding and DPI trimming

Inputs are made on the GPU from the seed: expression counts (zero-inflated negative
binomial, autocorrelated in pseudotime), independent draws from per-gene Dirichlet
distributions over the bins, or Markov chains over them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from tenex_b200 import TransferEntropyEngine
from tenex_b200.inference import NetWeaver
from tenex_b200.kernels import device as D
from tenex_b200.kernels import get_kernel
from tenex_b200.preprocess import remap_bins
from tenex_b200.result import TransferEntropyResult

DEVICE = "cuda"


def listed():
    return [
        # the smallest call: a marker panel, where launches and host waits count
        dict(name="compute_small", kind="compute", n=100, T=1000, tau=1),
        # a whole single-cell matrix of a few hundred cells, from host to host
        dict(name="compute_expression", kind="compute", n=3281, T=458, tau=1),
        # transcription factors as the only sources: the pair-list path, tau 2
        dict(name="compute_sources", kind="compute", n=2003, T=1001, tau=2, n_sources=150),
        # expression binarised at each gene's median, from host to host
        dict(name="compute_binarized", kind="compute", n=2000, T=5000, tau=1,
             binarization="median"),
        # a few thousand genes of few bins, autocorrelated: one TE matrix on the device
        dict(name="matrix_markov", kind="matrix", n=2000, T=5000, tau=1, values="markov",
             b_lo=2, b_hi=16, heavy=0.0),
        # finely binned genes: the largest histograms that need no coarsening
        dict(name="matrix_wide_bins", kind="matrix", n=2500, T=10000, tau=1, values="draws",
             b_lo=2, b_hi=32, heavy=0.0),
        # the largest call: every pair of 10,000 genes over 20,000 cells, uneven bins
        dict(name="matrix_uneven_large", kind="matrix", n=10000, T=20000, tau=1, values="draws",
             b_lo=2, b_hi=16, heavy=0.05),
        # a hundred thousand cells, few genes, an odd length
        dict(name="matrix_long_series", kind="matrix", n=301, T=101003, tau=1, values="draws",
             b_lo=2, b_hi=12, heavy=0.0),
        # binary bins on the tensor cores, device to device
        dict(name="binary_matrix", kind="binary", n=2000, T=5000, tau=1),
        # the significance test as it is, every surrogate computed for every pair
        dict(name="surrogate_full", kind="surrogate", n=1000, T=5000, tau=1, S=30, null="full"),
        # the same test with the learned null: prediction, then a list of pairs verified
        dict(name="surrogate_learned", kind="surrogate", n=2000, T=5000, tau=1, S=100,
             null="learned"),
        # the default network inference on a finished TE matrix
        dict(name="fdr_network", kind="fdr", n=5000, links=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["compute", "compute", "matrix", "matrix", "matrix", "binary", "surrogate",
                       "fdr"])
    tau = rng.choice([1, 1, 1, 2, 3])
    if kind == "compute":
        n, T = _log_int(rng, 30, 3500), _log_int(rng, 150, 6000)
        T = min(T, max(150, 10_000_000 // n))
        case = dict(kind=kind, n=n, T=T, tau=tau)
        form = rng.choice(["all", "all", "sources", "median", "mean"])
        if form == "sources":
            case["n_sources"] = max(1, n // rng.randint(8, 20))
        elif form != "all":
            case["binarization"] = form
        return case
    if kind == "matrix":
        n, T = _log_int(rng, 60, 6000), _log_int(rng, 300, 120_000)
        T = min(T, max(300, int(4e11 / n / n)))
        n = min(n, int(1.5e8 / T))
        b_hi = rng.choice([3, 4, 5, 6, 8, 10, 12, 16, 16, 24, 32])
        return dict(kind=kind, n=n, T=T, tau=tau, values=rng.choice(["draws", "markov"]), b_lo=2,
                    b_hi=b_hi, heavy=rng.choice([0.0, 0.0, 0.03, 0.08]))
    if kind == "binary":
        return dict(kind=kind, n=_log_int(rng, 80, 5000), T=_log_int(rng, 200, 12_000), tau=tau)
    if kind == "surrogate":
        return dict(kind=kind, n=_log_int(rng, 60, 1000), T=_log_int(rng, 300, 5000), tau=tau,
                    S=rng.randint(8, 30), null="full")
    return dict(kind=kind, n=_log_int(rng, 100, 5000), links=rng.choice([0, 0, 2000]))


# --------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed))


def _names(n):
    return np.array([f"G{i:05d}" for i in range(n)])


def _expression(case, seed):
    """float32 (n, T) log1p counts: a latent AR(1) per gene, Gamma-Poisson counts, 60%
    dropouts; one gene in twenty follows another with a lag of one."""
    n, T = case["n"], case["T"]
    g = _gen(seed)
    eps = torch.randn((T, n), generator=g, device=DEVICE) * 0.3
    z = torch.empty((T, n), device=DEVICE)
    z[0] = eps[0]
    for t in range(1, T):
        torch.add(eps[t], z[t - 1], alpha=0.9, out=z[t])
    k = n // 20
    if k:
        ids = torch.randperm(n, generator=g, device=DEVICE)[:2 * k]
        noise = torch.randn((T - 1, k), generator=g, device=DEVICE) * 0.3
        z[1:, ids[:k]] = 0.8 * z[:-1, ids[k:]] + noise
    mu = torch.exp(torch.randn(n, generator=g, device=DEVICE))
    gamma = -(torch.rand((T, n), generator=g, device=DEVICE).clamp_(min=1e-30).log_()
              + torch.rand((T, n), generator=g, device=DEVICE).clamp_(min=1e-30).log_())
    counts = torch.poisson(0.5 * gamma * mu * torch.exp(z), generator=g)
    counts[torch.rand((T, n), generator=g, device=DEVICE) < 0.6] = 0
    return torch.log1p(counts).t().contiguous().cpu().numpy()


def _bins(case, seed):
    """uint8 (n, T) raw bins on the device: per gene b bins with a Dirichlet(1)
    distribution, drawn independently ("draws": one gene in twenty repeats its last
    value half of the time) or as a chain that stays with probability 0.7 to 0.95
    ("markov"); a share `heavy` of genes has 64 to 256 bins."""
    n, T = case["n"], case["T"]
    g = _gen(seed)
    b = torch.randint(case["b_lo"], case["b_hi"] + 1, (n,), generator=g, device=DEVICE)
    heavy = torch.rand(n, generator=g, device=DEVICE) < case["heavy"]
    b = torch.where(heavy, torch.randint(64, 257, (n,), generator=g, device=DEVICE), b)
    wide = int(b.max())
    p = -torch.rand((n, wide), generator=g, device=DEVICE).clamp_(min=1e-30).log_()
    p *= torch.arange(wide, device=DEVICE)[None, :] < b[:, None]
    cum = torch.cumsum(p.double(), 1)
    cum = (cum / cum[:, -1:]).float()
    u = torch.rand(n, generator=g, device=DEVICE)
    if case["values"] == "markov":
        stay_p = 0.7 + 0.25 * u
    else:
        stay_p = torch.where(u < 0.05, 0.5, 0.0)
    out = torch.empty((n, T), dtype=torch.uint8, device=DEVICE)
    step = max(1, 40_000_000 // T)
    pos = torch.arange(T, device=DEVICE, dtype=torch.int32)
    for r in range(0, n, step):
        rows = slice(r, min(n, r + step))
        v = torch.searchsorted(cum[rows], torch.rand((rows.stop - r, T), generator=g,
                                                     device=DEVICE), right=True)
        v = torch.minimum(v, (b[rows] - 1)[:, None])
        stay = torch.rand((rows.stop - r, T), generator=g, device=DEVICE) < stay_p[rows, None]
        stay[:, 0] = False
        last = torch.where(stay, 0, pos).cummax(1).values
        out[rows] = torch.gather(v, 1, last.long()).to(torch.uint8)
    return out


def _binary(case, seed):
    """0/1 bins (n, T): two-state chains, stationary rate 0.05 to 0.5."""
    n, T = case["n"], case["T"]
    g = _gen(seed)
    pi = 0.05 + 0.45 * torch.rand(n, generator=g, device=DEVICE)
    stay_p = 0.7 + 0.25 * torch.rand(n, generator=g, device=DEVICE)
    v = (torch.rand((n, T), generator=g, device=DEVICE) < pi[:, None]).to(torch.uint8)
    stay = torch.rand((n, T), generator=g, device=DEVICE) < stay_p[:, None]
    stay[:, 0] = False
    pos = torch.arange(T, device=DEVICE, dtype=torch.int32)
    return torch.gather(v, 1, torch.where(stay, 0, pos).cummax(1).values.long())


def _dense(raw):
    """Dense relabelling of (n, T) uint8 bins in plain torch: bins, bin counts."""
    present = torch.zeros((raw.shape[0], 256), dtype=torch.int32, device=raw.device)
    present.scatter_(1, raw.long(), 1)
    rank = present.cumsum(1) - 1
    return torch.gather(rank, 1, raw.long()).to(torch.uint8), present.sum(1)


def _te_matrix(case, seed):
    """float32 (n, n) matrix as TE matrices come out: a plug-in bias that grows with
    both genes' bins, its spread, and 1% of pairs well above it."""
    n = case["n"]
    g = _gen(seed)
    src, tgt = (torch.randint(2, 17, (n,), generator=g, device=DEVICE).float() for _ in range(2))
    bias = (src[:, None] - 1) * tgt[None, :] * (tgt[None, :] - 1) * 1.5e-4
    m = bias * (1 + 0.1 * torch.randn((n, n), generator=g, device=DEVICE)).clamp_(min=0)
    edge = torch.rand((n, n), generator=g, device=DEVICE) < 0.01
    m = m + edge * 0.3 * torch.rand((n, n), generator=g, device=DEVICE)
    m.fill_diagonal_(0)
    return m.cpu().numpy()


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    if kind == "compute":
        state = dict(case=case, x=_expression(case, seed), names=_names(n), sources=None)
        if case.get("n_sources"):
            pick = np.random.default_rng(seed).permutation(n)[:case["n_sources"]]
            state["sources"] = state["names"][np.sort(pick)]
        return state
    if kind == "matrix":
        return dict(case=case, raw=_bins(case, seed))
    if kind == "binary":
        return dict(case=case, bins=D.pack_bins(_binary(case, seed), DEVICE, 2))
    if kind == "surrogate":
        bins, npv = _dense(_bins(dict(case, values="markov", b_lo=2, b_hi=16, heavy=0.0), seed))
        observed = _te_exact(bins, npv, case["tau"]).float().cpu().numpy()
        return dict(case=case, result=TransferEntropyResult(
            matrix=observed, variable_names=_names(n),
            bin_arrs=bins.cpu().numpy().astype(np.int8)[..., None],
            n_per_var=npv.cpu().numpy().astype(np.int32), b_max=int(npv.max()), tau=case["tau"],
            kernel="Full-SMEM"), edges=_Edges(n))
    return dict(case=case, matrix=_te_matrix(case, seed), names=_names(n), edges=_Edges(n),
                trimmed=_Edges(n))


class _Edges:
    """A network's edge list in arrays of one size for every network of n genes: its
    (source, target) rows and scores, then rows of -1 and scores of 0."""

    def __init__(self, n):
        room = max(1000, n * n // 10)
        self.pairs = np.full((room, 2), -1, np.int32)
        self.te = np.zeros(room, np.float32)

    def of(self, grn):
        self.pairs[:len(grn)] = grn.pairs
        self.te[:len(grn)] = grn.te
        return dict(pairs=self.pairs, te=self.te, count=len(grn))


# --------------------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    kind, tau = case["kind"], case.get("tau", 1)
    if kind == "compute":
        engine = TransferEntropyEngine(state["x"], state["names"], sources=state["sources"])
        res = engine.compute(accelerator="gpu", tau=tau, binarization=case.get("binarization"))
        return dict(matrix=res.matrix, bins=res.bin_arrs, n_per_var=res.n_per_var)
    if kind == "matrix":
        kernel = get_kernel("Adaptive-SMEM")
        bins, npv, b_max = remap_bins(state["raw"], 1, DEVICE)
        bins, npv, b_max = kernel.prepare(bins, npv, b_max, on_cuda=True, n_vars=case["n"],
                                          tau=tau)
        return kernel.compute_pairfree_device(bins, npv, b_max, tau, matrix=True)
    if kind == "binary":
        return get_kernel("GEMM-B2").compute_matrix_device(state["bins"], tau)
    if kind == "surrogate":
        res = NetWeaver(state["result"], fdr=0.05).infer(
            "surrogate_test", n_surrogates=case["S"], null=case["null"],
            block_length=_block_length(case))
        return dict(mean=res.mean_surrogate_te, std=res.std_surrogate_te,
                    effective=res.effective_te, p=res.p_values,
                    edges=state["edges"].of(res.grn))
    grn, trimmed = NetWeaver((state["matrix"], state["names"]), links=case["links"]).infer("fdr")
    return dict(edges=state["edges"].of(grn), trimmed=state["trimmed"].of(trimmed))


def _block_length(case):
    return 50 if case["T"] >= 1000 else max(2, int(math.sqrt(case["T"] - case["tau"])))


def work(case):
    """One histogram increment per sample of a pair (three multiply-adds per sample of
    a binary pair; one comparison per entry and mediator of a trimmed network's rows is
    not counted), inputs read once, results written once."""
    kind, n = case["kind"], case["n"]
    if kind == "fdr":
        return {"bytes": 4.0 * n * n, "flops": 4.0 * n * n}
    T, samples = case["T"], case["T"] - case["tau"]
    pairs = float(n) * (n - 1)
    if kind == "compute":
        out = 4.0 * n * n + 1.0 * n * T
        if case.get("n_sources"):
            pairs = float(case["n_sources"]) * (n - 1)
        ops = pairs * samples * (6 if case.get("binarization") else 1)
        return {"bytes": 4.0 * n * T + out, "flops": ops}
    if kind == "surrogate":
        passes = case["S"] if case["null"] == "full" else 1
        return {"bytes": 1.0 * n * T + 20.0 * n * n, "flops": pairs * samples * passes}
    return {"bytes": 1.0 * n * T + 4.0 * n * n,
            "flops": pairs * samples * (6 if kind == "binary" else 1)}


# --------------------------------------------------------------------------- 64 bits
def _te_exact(bins, npv, tau, sources=None):
    """float64 (n, n) TE, [source, target], of dense bins (n, T) in plain torch: joint
    counts as products of one-hot matrices (whole numbers, exact in float32), terms in
    float64. The diagonal, and rows of genes outside `sources`, are 0."""
    n, T = bins.shape
    dev = bins.device
    src = torch.arange(n, device=dev) if sources is None else torch.as_tensor(sources, device=dev)
    out = torch.zeros((n, n), dtype=torch.float64, device=dev)
    N = T - tau
    b_all = npv.tolist()
    tf32 = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = True  # 0 and 1 are exact in it
    try:
        group = max(1, int(6e9 / 4 / N / max(b_all)))
        for s0 in range(0, len(src), group):
            ids = src[s0:s0 + group]
            b = npv[ids].long()
            owner = torch.repeat_interleave(torch.arange(len(ids), device=dev), b)
            first = torch.cumsum(b, 0) - b
            value = torch.arange(len(owner), device=dev) - first[owner]
            hot = torch.empty((len(owner), N), device=dev)
            part = max(1, 200_000_000 // N)
            for r in range(0, len(owner), part):
                rows = slice(r, r + part)
                hot[rows] = bins[ids[owner[rows]], :N] == value[rows, None].to(torch.uint8)
            for t in range(n):
                bt = b_all[t]
                z = bins[t, tau:].long() * bt + bins[t, :N].long()
                state = torch.zeros((bt * bt, N), device=dev).scatter_(0, z[None, :], 1.0)
                out[ids, t] = _terms(state, hot, owner, len(ids), bt) / N
    finally:
        torch.backends.cuda.matmul.allow_tf32 = tf32
    out.fill_diagonal_(0)
    return out


def _terms(state, hot, owner, n_src, bt):
    c2a = state.sum(1, dtype=torch.float64)
    ratio = c2a.view(bt, bt).sum(0).expand(bt, bt) / c2a.view(bt, bt).clamp(min=1)
    total = torch.zeros(n_src, dtype=torch.float64, device=hot.device)
    rows = max(1, 60_000_000 // (bt * bt))
    for r in range(0, hot.shape[0], rows):
        c3 = (hot[r:r + rows] @ state.t()).double().view(-1, bt, bt)
        c2b = c3.sum(1, keepdim=True).clamp(min=1)
        term = torch.xlogy(c3, c3 * ratio / c2b).sum((1, 2)) / math.log(2.0)
        total.index_add_(0, owner[r:r + rows], term)
    return total


def _fsbwl(x):
    """Dense FSBW-L bins of float32 rows, in numpy's own float32 arithmetic (that is
    what defines them), at most 38 a gene (more are coarsened)."""
    bins = np.empty(x.shape, np.uint8)
    npv = np.empty(x.shape[0], np.int64)
    for i, row in enumerate(x):
        sd = row.std(ddof=1)
        sd = np.float32(1.0) if sd == 0 else sd
        raw = np.floor((row - (row.min() - np.float32(0.5) * sd)) / sd).astype(np.int64)
        values, rank = np.unique(np.maximum(raw, 0), return_inverse=True)
        b = len(values)
        bins[i], npv[i] = (rank, b) if b <= 38 else (rank * 38 // b, 38)
    return torch.from_numpy(bins).to(DEVICE), torch.from_numpy(npv).to(DEVICE)


def exact(case, seed):
    kind = case["kind"]
    if kind == "fdr" or case.get("null") == "learned":
        return None
    tau, n, T = case["tau"], case["n"], case["T"]
    if float(n) * n * T > 1.2e11:
        return None
    state = prepare(case, seed)
    if kind == "compute":
        x = state["x"]
        if case.get("binarization"):
            cut = np.median if case["binarization"] == "median" else np.mean
            hot = np.stack([row > cut(row) for row in x]).astype(np.uint8)
            bins = torch.from_numpy(hot).to(DEVICE)
            npv = torch.full((n,), 2, device=DEVICE)
        else:
            bins, npv = _fsbwl(x)
        src = None
        if state["sources"] is not None:
            src = np.searchsorted(state["names"], state["sources"])
        return dict(matrix=_te_exact(bins, npv, tau, src), bins=None, n_per_var=None)
    if kind == "matrix":
        bins, npv = _dense(state["raw"])
        over = npv > 38
        coarse = (bins.long() * 38 // npv[:, None]).to(torch.uint8)
        return _te_exact(torch.where(over[:, None], coarse, bins), npv.clamp(max=38), tau)
    if kind == "binary":
        bins = state["bins"]
        return _te_exact(bins.data[:, :T].contiguous(), torch.full((n,), 2, device=DEVICE), tau)
    # surrogate: the test's own permutations (a generator per surrogate, seeds 42 + k)
    res, S, length = state["result"], case["S"], _block_length(case)
    bins = torch.from_numpy(res.bin_arrs[..., 0].astype(np.uint8)).to(DEVICE)
    npv = torch.from_numpy(res.n_per_var).to(DEVICE)
    blocks = T // length
    g = torch.Generator(device=DEVICE)
    total = torch.zeros((n, n), dtype=torch.float64, device=DEVICE)
    square = torch.zeros_like(total)
    for k in range(S):
        g.manual_seed(42 + k)
        order = torch.argsort(torch.rand(n, blocks, device=DEVICE, generator=g), dim=1)
        head = bins[:, :blocks * length].view(n, blocks, length)
        head = torch.gather(head, 1, order[:, :, None].expand(-1, -1, length))
        te = _te_exact(torch.cat((head.reshape(n, -1), bins[:, blocks * length:]), 1), npv, tau)
        total += te
        square += te * te
    mean = total / S
    std = (square / S - mean * mean).clamp(min=0).sqrt()
    effective = torch.from_numpy(res.matrix).to(DEVICE).double() - mean
    p = 0.5 * torch.special.erfc(effective / std.clamp(min=1e-12) / math.sqrt(2.0))
    p.fill_diagonal_(1.0)
    return dict(mean=mean, std=std, effective=effective, p=p, edges=None)
