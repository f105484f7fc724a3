"""Timed workloads of the GPU sampler, through the package's public entry points.

A case is what a user's program runs over and over: iterations of a Gibbs
chain with the read-back of a sample (`Chain`, `Batch`, `Multi`), the packing
of a PLINK BED payload, or genetic values from marker effects.  Sizes follow
the benchmark's configurations (dense N = 2,000 x M = 5,000, ragged N = 20,000 x
M = 50,000, dense N = M = 100,000 with two groups, batched chains at N = 50,000,
independent regressions of uneven sizes) with odd and small sizes beside them.

`prepare` makes genotypes and phenotypes on the GPU from the seed alone and
hands over a chain that is ready to iterate: freshly initialised (burn-in,
where many markers change per sweep) or resumed from the state of a chain that
has left its burn-in (about one marker in a hundred carries an effect).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from bayesrrcmd_gb300 import gpu

KINDS = {"dense": gpu.KIND_DENSE, "ragged": gpu.KIND_RAGGED, "eigen": gpu.KIND_EIGEN}
S_ONE = [[0.01, 0.001, 0.0001]]                  # the reference's default mixture
S_TWO = [[0.01, 0.001, 0.0001], [0.1, 0.01]]     # the benchmark's two groups


def _chain(name, kind, form, N, M, groups=1, missing=0.0, p_lo=0.05, rare=False, iters=1, resumed=False, tokens=0):
    c = dict(what="chain", kind=kind, form=form, N=N, M=M, groups=groups, missing=missing, p_lo=p_lo, rare=rare,
             iters=iters, resumed=resumed, tokens=tokens)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # a pilot run on a few hundred people and markers: launches and latency
        _chain("dense_fp64_tiny", "dense", "fp64", 503, 401),
        # a small candidate-region study, the default (FP64) form, burn-in
        _chain("dense_fp64_small", "dense", "fp64", 2_000, 5_000),
        # the same study in the FP32-compensated form, saving every fifth sample
        _chain("dense_fp32c_small", "dense", "fp32c", 2_000, 5_000, iters=5, resumed=True),
        # a cohort with imputation gaps, odd sizes, two groups
        _chain("dense_fp32c_missing", "dense", "fp32c", 20_011, 30_001, groups=2, missing=0.01, iters=5, resumed=True),
        # the benchmark's size in the default form
        _chain("dense_fp64_large", "dense", "fp64", 100_000, 100_000, groups=2, p_lo=0.01, resumed=True),
        # the benchmark's chosen form at its size
        _chain("dense_fp32c_large", "dense", "fp32c", 100_000, 100_000, groups=2, p_lo=0.01, iters=2, resumed=True),
        # the sparse benchmark in the default form, burn-in
        _chain("ragged_fp64", "ragged", "fp64", 20_000, 50_000, missing=0.005, p_lo=0.005, rare=True),
        # the sparse benchmark in the compensated form after the burn-in
        _chain("ragged_fp32c", "ragged", "fp32c", 20_000, 50_000, missing=0.005, p_lo=0.005, rare=True, iters=5,
               resumed=True),
        # the Eigen marker kind on an odd-sized panel
        _chain("eigen_fp64", "eigen", "fp64", 9_973, 12_345, missing=0.02, p_lo=0.005, rare=True, resumed=True),
        # 64 phenotypes of one cohort swept together
        dict(name="batch_64", what="batch", chains=64, N=50_000, M=40_000, p_lo=0.01, iters=5),
        # regressions of different sizes in one launch (dense and ragged)
        dict(name="uneven_12", what="uneven", count=12, N_lo=1_000, N_hi=50_000, M_lo=2_000, M_hi=40_000,
             missing=0.01, iters=1),
        # reading a BED file's payload into standardised markers
        dict(name="pack_ragged", what="pack", kind="ragged", N=20_011, M=20_000, missing=0.005, p_lo=0.005, rare=True),
    ]


def _log_int(rng, lo, hi):
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return min(hi, max(lo, v | 1 if rng.random() < 0.5 else v))


def draw(rng):
    r = rng.random()
    if r < 0.72:
        kind = rng.choice(["dense", "dense", "ragged", "eigen"])
        form = rng.choice(["fp64", "fp32c"])
        N = _log_int(rng, 300, 100_000)
        M = _log_int(rng, 400, 100_000 if kind == "dense" else 50_000)
        while N * M > 4_000_000_000:
            M = max(400, M // 2 + 1)
        return _chain(None, kind, form, N, M, groups=rng.choice([1, 2]), missing=rng.choice([0.0, 0.005, 0.02]),
                      p_lo=round(rng.uniform(0.03, 0.1), 3), rare=rng.random() < 0.3,
                      iters=min(rng.choice([1, 2, 5]), max(1, 100_000 // M)),
                      resumed=rng.random() < 0.6,
                      tokens=rng.choice([0, 0, 20]) if form == "fp64" else 0)
    if r < 0.82:
        return dict(what="batch", chains=rng.choice([32, 64]), N=_log_int(rng, 2_000, 50_000),
                    M=_log_int(rng, 1_000, 40_000), p_lo=round(rng.uniform(0.02, 0.1), 3), iters=rng.choice([1, 2, 5]))
    if r < 0.9:
        return dict(what="uneven", count=rng.randint(3, 12), N_lo=1_000, N_hi=_log_int(rng, 5_000, 50_000),
                    M_lo=1_000, M_hi=_log_int(rng, 5_000, 40_000), missing=rng.choice([0.0, 0.01]), iters=1)
    if r < 0.95:
        return dict(what="pack", kind=rng.choice(["dense", "ragged", "eigen"]), N=_log_int(rng, 1_000, 50_000),
                    M=_log_int(rng, 1_000, 8_000), missing=rng.choice([0.0, 0.01]), p_lo=0.03, rare=False)
    N = _log_int(rng, 2_000, 100_000)
    return dict(what="predict", kind=rng.choice(["dense", "ragged"]), N=N,
                M=min(_log_int(rng, 2_000, 40_000), 2_000_000_000 // N), effects=_log_int(rng, 100, 2_000),
                missing=rng.choice([0.0, 0.01]), p_lo=0.03, rare=False)


# ---------------------------------------------------------------------------
# Inputs.

def _rng(seed, salt):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, salt])


def _bed(N, M, seed, salt, p_lo, missing, rare=False, p_hi=0.5):
    """M x ceil(N/4) bytes of PLINK 2-bit genotypes on the GPU: allele
    frequencies uniform in [p_lo, p_hi], or log-uniform (`rare`)."""
    g = torch.Generator(device="cuda").manual_seed((int(seed) * 1_000_003 + salt) & 0x7FFFFFFF)
    nb = (N + 3) // 4
    out = torch.empty((M, nb), dtype=torch.uint8, device="cuda")
    p = torch.rand(M, generator=g, device="cuda", dtype=torch.float64)
    lo = max(p_lo, 8.0 / N)     # a marker seen in one person at least
    p = torch.exp(math.log(lo) + p * (math.log(p_hi) - math.log(lo))) if rare else lo + p * (p_hi - lo)
    step = max(1, min(M, 60_000_000 // (4 * nb)))
    for a in range(0, M, step):
        q = p[a:a + step].float()[:, None]
        u = torch.rand((q.shape[0], 4 * nb), generator=g, device="cuda")
        code = torch.full_like(u, 3, dtype=torch.uint8)
        code[u < q * (2 - q)] = 2
        code[u < q * q] = 0
        if missing > 0:
            code[torch.rand(u.shape, generator=g, device="cuda") < missing] = 1
        code[:, N:] = 0
        code = code.view(-1, nb, 4)
        out[a:a + step] = code[..., 0] | (code[..., 1] << 2) | (code[..., 2] << 4) | (code[..., 3] << 6)
    return out


_VALUE = {"g": (2.0, 0.0, 1.0, 0.0), "m": (0.0, 1.0, 0.0, 0.0)}


def _decode(bed, N, which="g"):
    """Genotypes (missing 0) or the missing indicator of some markers, float64."""
    lut = torch.tensor(_VALUE[which], dtype=torch.float64, device=bed.device)
    table = torch.stack([lut[(torch.arange(256, device=bed.device) >> (2 * k)) & 3] for k in range(4)], 1)
    return table[bed.long()].view(bed.shape[0], -1)[:, :N]


def _columns(bed, N, kind):
    """(D, W, mean, sd, zsum) of some markers: the dot product reads D, the
    residual moves along W.  Dense markers are centred and scaled columns with
    the missing genotypes at the mean; the sparse kinds hold genotype values
    with mean and sd aside and leave missing genotypes unmoved."""
    g, m = _decode(bed, N), _decode(bed, N, "m")
    if kind == "dense":
        mean = g.sum(1, keepdim=True) / (N - m.sum(1, keepdim=True))
        v = g + m * mean
        v = v - v.mean(1, keepdim=True)
        x = v / torch.sqrt((v * v).sum(1, keepdim=True) / (N - 1.0))
        return x, x, None, None, None
    mean = g.sum(1, keepdim=True) / N
    z = g + m * mean if kind == "eigen" else g
    zsum, sq = z.sum(1, keepdim=True), (z * z).sum(1, keepdim=True)
    sd = torch.sqrt((sq - 2.0 * mean * zsum + N * mean * mean) / (N - 1.0))
    w = (g - mean * (1.0 - m)) / sd
    return z, w, mean[:, 0], sd[:, 0], zsum[:, 0]


def _phenotype(bed, N, M, kind, n_causal, h2, rng):
    """Float32 phenotype of n_causal standardised markers, with the effects."""
    causal = np.sort(rng.choice(M, n_causal, replace=False))
    b = rng.normal(0.0, math.sqrt(h2 / n_causal), n_causal)
    gv = torch.zeros(N, dtype=torch.float64, device="cuda")
    step = max(1, 20_000_000 // N)
    for a in range(0, n_causal, step):
        _, w, _, _, _ = _columns(bed[torch.from_numpy(causal[a:a + step]).cuda()], N, kind)
        gv += torch.from_numpy(b[a:a + step]).cuda() @ w
    gv = gv.cpu().numpy()
    y = (gv + rng.normal(0.0, math.sqrt(1.0 - h2), N)).astype(np.float32)
    return y, causal, b, gv


def _standardise(y):
    y = y.astype(np.float64)
    d = y - y.mean()
    return d / math.sqrt((d * d).sum() / (len(y) - 1))


def _mixture(case):
    return S_TWO if case.get("groups", 1) == 2 else S_ONE


def _groups(M, n_groups):
    return (np.arange(M) % n_groups).astype(np.int32)


def _resumed(case, y, causal, b, gv):
    """The state of a chain past its burn-in: the causal effects found, the
    residual that is left, and variances and mixture weights to match."""
    S, M, N = _mixture(case), case["M"], case["N"]
    ys = y.astype(np.float64)
    sd = math.sqrt(((ys - ys.mean()) ** 2).sum() / (N - 1))
    beta = np.zeros(M)
    comp = np.zeros(M, np.int32)
    beta[causal] = b / sd
    group = _groups(M, len(S))
    sigma_g = np.zeros(len(S))
    pi = np.zeros((len(S), gpu.MAX_K))
    for q, s in enumerate(S):
        mine = causal[group[causal] == q]
        # a tiny panel may leave a group without causal markers
        total = max(float((beta[mine] ** 2).sum()), 0.05 / len(S))
        sigma_g[q] = total
        comp[mine] = 1 + np.abs(np.log(np.maximum(beta[mine, None] ** 2, 1e-30) / (total * np.array(s)))).argmin(1)
        in_group = np.count_nonzero(group == q)
        pi[q, 1:len(s) + 1] = [(np.count_nonzero(comp[mine] == k + 1) + 1.0) / (in_group + len(s) + 1)
                               for k in range(len(s))]
        pi[q, 0] = 1.0 - pi[q].sum()
    eps = _standardise(y) - (gv - gv.mean()) / sd
    return dict(beta=beta, comp=comp, acum=np.full(M, 0.5), eps=eps, mu=0.0,
                sigmaE=float((eps * eps).sum() / N), epsSum=float(eps.sum()), sigmaG=sigma_g, pi=pi, iteration=0)


def _causal_count(M):
    return max(2, M // 100 if M <= 50_000 else 1_000)


def _chain_inputs(case, seed):
    N, M = case["N"], case["M"]
    bed = _bed(N, M, seed, 1, case["p_lo"], case["missing"], case["rare"])
    y, causal, b, gv = _phenotype(bed, N, M, case["kind"], _causal_count(M), 0.45, _rng(seed, 2))
    return bed, y, (_resumed(case, y, causal, b, gv) if case["resumed"] else None)


def _batch_inputs(case, seed):
    N, M = case["N"], case["M"]
    bed = _bed(N, M, seed, 1, case["p_lo"], 0.0)
    rng = _rng(seed, 2)
    y = np.stack([_phenotype(bed, N, M, "dense", _causal_count(M) // 2 + 1, rng.uniform(0.1, 0.7), rng)[0]
                  for _ in range(case["chains"])])
    return bed, y


def _uneven_sizes(case):
    """Sizes spread over the case's ranges, large N beside small M and the reverse."""
    n = case["count"]
    t = (np.arange(n) + 0.5) / n
    s = (np.arange(n) * 5 % n + 0.5) / n
    N = np.exp(math.log(case["N_lo"]) + t * math.log(case["N_hi"] / case["N_lo"])).astype(int) | 1
    M = np.exp(math.log(case["M_lo"]) + s * math.log(case["M_hi"] / case["M_lo"])).astype(int)
    return [(int(a), int(b)) for a, b in zip(N, M)]


def _uneven_inputs(case, seed):
    out = []
    for i, (N, M) in enumerate(_uneven_sizes(case)):
        # every third panel is sequenced (rare variants, index lists), the others are chips
        kind = "ragged" if i % 3 == 2 else "dense"
        bed = _bed(N, M, seed, 10 + i, 0.02, case["missing"], rare=kind == "ragged")
        y, _, _, _ = _phenotype(bed, N, M, kind, max(2, M // 200), 0.4, _rng(seed, 100 + i))
        out.append((kind, N, M, bed, y))
    return out


def _config(case, seed):
    return gpu.ChainConfig(N=case["N"], M=case["M"], kind=KINDS[case["kind"]],
                           form=gpu.FORM_FP64 if case["form"] == "fp64" else gpu.FORM_FP32C, S=_mixture(case),
                           seed=int(seed) & 0x7FFFFFFF, refresh_every=0 if case["form"] == "fp64" else 50,
                           async_batch=case["tokens"])


def prepare(case, seed):
    if case["what"] == "chain":
        bed, y, state = _chain_inputs(case, seed)
        ch = gpu.Chain(_config(case, seed))
        torch.cuda.synchronize()
        ch.pack_bed_device(bed.data_ptr(), bed.numel())
        ch.set_groups(_groups(case["M"], case["groups"]))
        ch.set_phenotype(y)
        if state is None:
            ch.init()
        else:
            ch.set_state(state)
        return dict(case=case, chain=ch)
    if case["what"] == "batch":
        bed, y = _batch_inputs(case, seed)
        b = gpu.Batch(gpu.ChainConfig(N=case["N"], M=case["M"], form=gpu.FORM_FP32C, S=S_ONE,
                                      seed=int(seed) & 0x7FFFFFFF), case["chains"])
        torch.cuda.synchronize()
        b.pack_bed_device(bed.data_ptr(), bed.numel())
        b.set_phenotypes(y)
        b.init()
        return dict(case=case, batch=b)
    if case["what"] == "uneven":
        parts = _uneven_inputs(case, seed)
        m = gpu.Multi([gpu.ChainConfig(N=N, M=M, kind=KINDS[kind], form=gpu.FORM_FP32C, S=S_ONE,
                                       seed=int(seed) & 0x7FFFFFFF, chain=i, refresh_every=50)
                       for i, (kind, N, M, _, _) in enumerate(parts)])
        torch.cuda.synchronize()
        for i, (_, _, _, bed, y) in enumerate(parts):
            m.pack_bed_device(i, bed.data_ptr(), bed.numel())
            m.set_phenotype(i, y)
        m.init()
        m.tune(2)
        return dict(case=case, multi=m)
    bed = _bed(case["N"], case["M"], seed, 1, case["p_lo"], case["missing"], case["rare"])
    if case["what"] == "pack":
        return dict(case=case, bed=bed.cpu().numpy())
    ch = gpu.Chain(gpu.ChainConfig(N=case["N"], M=case["M"], kind=KINDS[case["kind"]], S=S_ONE))
    torch.cuda.synchronize()
    ch.pack_bed_device(bed.data_ptr(), bed.numel())
    idx, b = _effects(case, seed)
    return dict(case=case, chain=ch, idx=idx, b=b)


def _effects(case, seed):
    rng = _rng(seed, 3)
    n = min(case["effects"], case["M"])
    return (np.sort(rng.choice(case["M"], n, replace=False)).astype(np.uint32), rng.normal(0.0, math.sqrt(0.4 / n), n))


def run(state):
    case = state["case"]
    if case["what"] == "chain":
        state["chain"].iterate(case["iters"])
        return state["chain"].state()
    if case["what"] == "batch":
        state["batch"].iterate(case["iters"])
        rows = [state["batch"].state(c) for c in range(case["chains"])]
        return {k: np.stack([r[k] for r in rows]) for k in rows[0]}
    if case["what"] == "uneven":
        state["multi"].iterate(case["iters"])
        # one array per quantity, the instances one after the other
        rows = [state["multi"].state(i) for i in range(case["count"])]
        return {k: np.concatenate([np.ravel(r[k]) for r in rows]) for k in rows[0]}
    if case["what"] == "pack":
        with gpu.Chain(gpu.ChainConfig(N=case["N"], M=case["M"], kind=KINDS[case["kind"]], S=S_ONE)) as ch:
            ch.pack_bed(state["bed"])
            table, counts = ch.marker_table()
            return dict(table=table, counts=counts)
    return state["chain"].xbeta(state["idx"], state["b"])


def work(case):
    """Per sweep every genotype is read once (2 bits each) and enters one dot
    product (a multiply and an add); the state is written and read back once."""
    def state(N, M):
        return M * 20 + N * 8

    if case["what"] == "chain":
        N, M, it = case["N"], case["M"], case["iters"]
        return dict(bytes=it * N * M / 4 + state(N, M), flops=2.0 * it * N * M)
    if case["what"] == "batch":
        N, M, it, C = case["N"], case["M"], case["iters"], case["chains"]
        return dict(bytes=it * N * M / 4 + C * state(N, M), flops=2.0 * it * N * M * C)
    if case["what"] == "uneven":
        g = sum(N * M for N, M in _uneven_sizes(case))
        return dict(bytes=case["iters"] * g / 4 + sum(state(N, M) for N, M in _uneven_sizes(case)),
                    flops=2.0 * case["iters"] * g)
    if case["what"] == "pack":
        return dict(bytes=case["N"] * case["M"] / 4 + case["M"] * 64, flops=float(case["N"]) * case["M"])
    return dict(bytes=case["effects"] * case["N"] / 4 + case["N"] * 8, flops=2.0 * case["effects"] * case["N"])


# ---------------------------------------------------------------------------
# The same answers in 64 bits from plain numpy and torch.

def _philox(c0, c1, c2, c3, k0, k1):
    """Philox4x32-10 (Salmon et al. 2011) over arrays of counters."""
    c = [np.asarray(x, np.uint64) for x in np.broadcast_arrays(c0, c1, c2, c3)]
    k0, k1, low = np.uint64(k0), np.uint64(k1), np.uint64(0xFFFFFFFF)
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ k0, p1 & low, (p0 >> np.uint64(32)) ^ c[3] ^ k1, p0 & low]
        k0, k1 = (k0 + np.uint64(0x9E3779B9)) & low, (k1 + np.uint64(0xBB67AE85)) & low
    return c


def _u53(a, b):
    return ((a >> np.uint64(5)).astype(np.float64) * 67108864.0 + (b >> np.uint64(6)).astype(np.float64) + 0.5) / 2.0 ** 53


def _normal(v1, v2):
    return np.sqrt(-2.0 * np.log(v1)) * np.cos(6.283185307179586 * v2)


class _Stream:
    """The draws of one chain, each a function of (seed, chain, index, iteration)."""
    INIT, MU, MARKER, PERM, SIGMA_E, SIGMA_G, PI = 1, 2, 3, 4, 5, 6, 7

    def __init__(self, seed, chain):
        self.key = (int(seed) & 0xFFFFFFFF, int(chain))

    def block(self, idx, it, purpose, sub=0):
        return _philox(idx, it, purpose, sub, *self.key)

    def marker(self, it, M):
        j = np.arange(M)
        b, c = self.block(j, it, self.MARKER), self.block(j, it, self.MARKER, 1)
        return _u53(b[0], b[1]), _normal(_u53(b[2], b[3]), _u53(c[0], c[1]))

    def order(self, it, M):
        b = self.block(np.arange(M), it, self.PERM)
        r = ((b[0] << np.uint64(32)) | b[1]).tolist()
        perm = list(range(M))
        for i in range(M - 1, 0, -1):
            j = (r[i] * (i + 1)) >> 64
            perm[i], perm[j] = perm[j], perm[i]
        return np.array(perm)

    def mu(self, it):
        b = self.block(0, it, self.MU)
        return float(_normal(_u53(b[0], b[1]), _u53(b[2], b[3])))

    def gamma(self, it, purpose, sub, shape):
        a = shape + 1.0 if shape < 1.0 else shape
        d = a - 1.0 / 3.0
        c = 1.0 / math.sqrt(9.0 * d)
        for t in range(1024):
            b, e = self.block(t, it, purpose, sub), self.block(t, it, purpose, sub | 0x80000000)
            x = float(_normal(_u53(b[0], b[1]), _u53(b[2], b[3])))
            v = 1.0 + c * x
            if v <= 0.0:
                continue
            v = v * v * v
            u = float(_u53(e[0], e[1]))
            if u < 1.0 - 0.0331 * x ** 4 or math.log(u) < 0.5 * x * x + d * (1.0 - v + math.log(v)):
                return d * v * (float(_u53(e[2], e[3])) ** (1.0 / shape) if shape < 1.0 else 1.0)
        raise ValueError("no gamma draw")

    def inv_chisq(self, it, purpose, sub, dof, scale):
        return 0.5 * dof * scale / self.gamma(it, purpose, sub, 0.5 * dof)


class _Exact:
    """BayesR chains on shared markers, marker by marker in 64 bits; blocks of
    64 markers share one product with the residuals, corrected after every
    change by the markers' products with each other."""
    PRIOR = 1e-4

    def __init__(self, bed, N, M, kind, S, group, ys, seed, chains, state=None, tokens=0):
        self.bed, self.N, self.M, self.kind, self.S, self.group, self.tokens = bed, N, M, kind, S, group, tokens
        self.streams = [_Stream(seed, c) for c in chains]
        C, G = len(chains), len(S)
        self.beta, self.comp, self.acum = np.zeros((M, C)), np.zeros((M, C), np.int32), np.zeros((M, C))
        self.eps = torch.from_numpy(np.stack([_standardise(y) for y in ys], 1)).cuda()
        self.mu = np.zeros(C)
        self.sigma_g = np.array([[float(_u53(*s.block(g, 0, s.INIT)[:2])) for s in self.streams] for g in range(G)])
        self.pi = np.zeros((G, gpu.MAX_K, C))
        for g, s in enumerate(S):
            self.pi[g, 0] = 0.5
            self.pi[g, 1:len(s) + 1] = 0.5 / (len(s) + 1)
        if state is not None:
            for name in ("beta", "comp", "acum"):
                getattr(self, name)[:, 0] = state[name]
            self.eps = torch.from_numpy(state["eps"][:, None].copy()).cuda()
            self.sigma_g[:, 0], self.pi[:, :, 0] = state["sigmaG"], state["pi"]
        e = self.eps.cpu().numpy()
        self.sigma_e = (e * e).sum(0) / N * (0.5 if state is None else 1.0)
        self.eps_sum = e.sum(0)
        self.iteration = 0

    def _pick(self, j, num, u, z, const):
        """One marker's component and effect for every chain."""
        K, log_c, inv_den, h, sd = const
        C = len(num)
        if C == 1:
            n2 = float(num[0]) ** 2
            L = [log_c[0][0]] + [log_c[k][0] + n2 * h[k][0] for k in range(1, K)]

            def prob(k):
                if any(abs(x - L[k]) > 700 for x in L[1:]):
                    return 0.0
                return 1.0 / sum(math.exp(x - L[k]) for x in L)

            acc = a0 = prob(0)
            got = -1
            for k in range(K):
                if u[j, 0] <= acc:
                    got = k
                    break
                if k + 1 < K:
                    acc += prob(k + 1)
            old = self.beta[j, 0]
            new = old if got < 0 else 0.0 if got == 0 else z[j, 0] * sd[got][0] + num[0] * inv_den[got][0]
            self.acum[j, 0] = a0 if not self.tokens else self.acum[j, 0]
            if got >= 0:
                self.comp[j, 0] = got
            self.chosen[j, 0] = got >= 0
            self.beta[j, 0] = new
            return np.array([old - new])
        L = np.concatenate([log_c[:1], log_c[1:] + num * num * h[1:]])
        with np.errstate(over="ignore"):
            P = 1.0 / np.exp(L[None, :, :] - L[:, None, :]).sum(1)
        P[(np.abs(L[None, 1:, :] - L[:, None, :]) > 700).any(1)] = 0.0
        cum = np.cumsum(P, 0)
        hit = u[j] <= cum
        got = np.where(hit.any(0), hit.argmax(0), -1)
        at = np.arange(C)
        new = np.where(got > 0, z[j] * sd[got, at] + num * inv_den[got, at], np.where(got == 0, 0.0, self.beta[j]))
        old = self.beta[j].copy()
        self.acum[j] = P[0]
        self.comp[j] = np.where(got >= 0, got, self.comp[j])
        self.chosen[j] = got >= 0
        self.beta[j] = new
        return old - new

    def iterate(self):
        N, M, it, S = self.N, self.M, self.iteration, self.S
        sparse = self.kind != "dense"
        self.eps += torch.from_numpy(self.mu).cuda()
        total = self.eps.sum(0).cpu().numpy()
        if sparse:
            self.eps_sum = self.eps_sum + self.mu * N
            total = self.eps_sum
        self.mu = total / N + np.sqrt(self.sigma_e / N) * np.array([s.mu(it) for s in self.streams])
        self.eps -= torch.from_numpy(self.mu).cuda()
        if sparse:
            self.eps_sum = self.eps_sum - self.mu * N
        draws = [s.marker(it, M) for s in self.streams]
        u, z = np.stack([d[0] for d in draws], 1), np.stack([d[1] for d in draws], 1)
        order = self.streams[0].order(it, M)
        self.chosen = np.zeros((M, len(self.streams)), bool)
        const = []
        for g, s in enumerate(S):
            K = len(s) + 1
            cva = np.concatenate([[1.0], s])[:, None]
            denom = (N - 1.0) + self.sigma_e / self.sigma_g[g] / cva
            log_c = np.log(self.pi[g, :K]) - 0.5 * np.log(self.sigma_g[g] / self.sigma_e * (N - 1.0) * cva + 1.0)
            log_c[0] = np.log(self.pi[g, 0])
            const.append((K, log_c, 1.0 / denom, 0.5 / denom / self.sigma_e, np.sqrt(self.sigma_e / denom)))
        width = self.tokens or 64
        for q in range(0, M, width):
            block = order[q:q + width]
            D, W, mean, sd, zsum = _columns(self.bed[torch.from_numpy(block).cuda()], N, self.kind)
            dots = (D @ self.eps).cpu().numpy()
            G = (D @ W.T).cpu().numpy()
            if sparse:
                mean, sd, zsum = mean.cpu().numpy(), sd.cpu().numpy(), zsum.cpu().numpy()
            delta = np.zeros((len(block), len(self.streams)))
            sum0 = self.eps_sum
            for t, j in enumerate(block):
                dot = dots[t] if self.tokens else dots[t] + G[t, :t] @ delta[:t]
                if sparse:
                    dot = (dot - mean[t] * (sum0 if self.tokens else self.eps_sum)) / sd[t]
                delta[t] = self._pick(j, dot + self.beta[j] * (N - 1.0), u, z, const[self.group[j]])
                if sparse:
                    self.eps_sum = self.eps_sum + delta[t] * (zsum[t] - mean[t] * N) / sd[t]
            self.eps += W.T @ torch.from_numpy(delta).cuda()
        e2 = (self.eps * self.eps).sum(0).cpu().numpy()
        p = self.PRIOR
        for c, s in enumerate(self.streams):
            self.sigma_e[c] = s.inv_chisq(it, s.SIGMA_E, 0, p + N, (e2[c] + p * p) / (p + N))
            for g in range(len(S)):
                K = const[g][0]
                mine = (self.group == g) & self.chosen[:, c]
                v = np.bincount(self.comp[mine, c], minlength=K).astype(np.float64)
                m0 = float(v[1:].sum())
                bsq = float((self.beta[mine & (self.comp[:, c] > 0), c] ** 2).sum())
                self.sigma_g[g, c] = s.inv_chisq(it, s.SIGMA_G, g, p + m0, (bsq * m0 + p * p) / (p + m0))
                d = np.array([s.gamma(it, s.PI, g * 256 + k, v[k] + 1.0) for k in range(K)])
                self.pi[g, :K, c] = d / d.sum()
        self.iteration += 1

    def rows(self):
        eps = self.eps.cpu().numpy()
        return [dict(beta=self.beta[:, c].copy(), comp=self.comp[:, c].copy(), acum=self.acum[:, c].copy(),
                     eps=eps[:, c].copy(), mu=float(self.mu[c]), sigmaE=float(self.sigma_e[c]),
                     epsSum=float(self.eps_sum[c]) if self.kind != "dense" else None, sigmaG=self.sigma_g[:, c].copy(),
                     pi=self.pi[:, :, c].copy(), iteration=self.iteration) for c in range(len(self.streams))]


def _seconds(N, M, iters, chains=1):
    """Rough cost of the 64-bit replay."""
    return iters * M * (3e-5 + (8e-5 if chains > 1 else 0.0) + 5e-10 * N * (1 + chains / 32))


def exact(case, seed):
    key = int(seed) & 0x7FFFFFFF
    if case["what"] == "chain":
        N, M = case["N"], case["M"]
        if _seconds(N, M, case["iters"]) > 20:
            return None
        bed, y, state = _chain_inputs(case, seed)
        ex = _Exact(bed, N, M, case["kind"], _mixture(case), _groups(M, case["groups"]), [y], key, [0], state,
                    case["tokens"])
        for _ in range(case["iters"]):
            ex.iterate()
        return ex.rows()[0]
    if case["what"] == "batch":
        N, M, C = case["N"], case["M"], case["chains"]
        if _seconds(N, M, case["iters"], C) > 20:
            return None
        bed, y = _batch_inputs(case, seed)
        ex = _Exact(bed, N, M, "dense", S_ONE, _groups(M, 1), list(y), key, list(range(C)))
        for _ in range(case["iters"]):
            ex.iterate()
        rows = ex.rows()
        return {k: None if rows[0][k] is None else np.stack([r[k] for r in rows]) for k in rows[0]}
    if case["what"] == "uneven":
        # choosing the round widths runs five iterations of every chain
        iters = 5 + case["iters"]
        if sum(_seconds(N, M, iters) for N, M in _uneven_sizes(case)) > 20:
            return None
        rows = []
        for i, (kind, N, M, bed, y) in enumerate(_uneven_inputs(case, seed)):
            ex = _Exact(bed, N, M, kind, S_ONE, _groups(M, 1), [y], key, [i])
            for _ in range(iters):
                ex.iterate()
            rows += ex.rows()
        return {k: None if any(r[k] is None for r in rows) else np.concatenate([np.ravel(r[k]) for r in rows])
                for k in rows[0]}
    N, M = case["N"], case["M"]
    bed = _bed(N, M, seed, 1, case["p_lo"], case["missing"], case["rare"])
    if case["what"] == "predict":
        idx, b = _effects(case, seed)
        out = torch.zeros(N, dtype=torch.float64, device="cuda")
        step = max(1, 20_000_000 // N)
        for a in range(0, len(idx), step):
            _, w, _, _, _ = _columns(bed[torch.from_numpy(idx[a:a + step].astype(np.int64)).cuda()], N, case["kind"])
            out += torch.from_numpy(b[a:a + step]).cuda() @ w
        return out.cpu().numpy()
    if case["kind"] == "dense":
        table = np.zeros((M, 4))
        step = max(1, 20_000_000 // N)
        for a in range(0, M, step):
            g, m = _decode(bed[a:a + step], N), _decode(bed[a:a + step], N, "m")
            nm, q = m.sum(1), g.sum(1)
            mean = q / (N - nm)
            col = (q + nm * mean) / N
            v = g + m * mean[:, None] - col[:, None]
            s = 1.0 / torch.sqrt((v * v).sum(1) / (N - 1.0))
            table[a:a + step] = torch.stack([(2.0 - col) * s, (mean - col) * s, (1.0 - col) * s, -col * s], 1).cpu().numpy()
        return dict(table=table, counts=None)
    rows = []
    step = max(1, 20_000_000 // N)
    for a in range(0, M, step):
        z, _, mean, sd, zsum = _columns(bed[a:a + step], N, case["kind"])
        rows.append(torch.stack([mean, sd, (z * z).sum(1), zsum], 1).cpu().numpy())
    return dict(table=np.concatenate(rows), counts=None)
