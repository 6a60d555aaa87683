"""Timed cases of the package: what a program that uses it calls, over the sizes it meets.

listed() names the cases, draw() gives more of the same ranges, prepare() makes a case's inputs
from a seed (and loads them where the program holds them on the GPU before the call), run() is one
pass through the public entry points and returns all they compute, work() is what the pass cannot
do without, and exact() the same results from plain torch in 64 bits.

Kinds:
  pca      a top-k PCA (rsvd) of a genotype panel: Halko (svd=1) or window-based (svd=2), on
           genotypes already loaded ("resident"), from host records through upload, shuffle and
           PCA ("whole"), or streamed from host memory ("streamed")
  emu      EMU on a panel with much missing data: the first EM iteration and the final
           standardised PCA (emu_loop with maxiter=1: three RSVDs, two imputations)
  pcangsd  PCAngsd on genotype likelihoods: allele frequencies, the initial posterior, a PCA, one
           EM update and the PCA after it
  grm      the PCAngsd covariance matrix from final factors
  ld       r2 of every SNP pair within a window, genotypes projected off the top PCs or not
  gram     Z (Z^T X), the matrix operation of the Arnoldi / Lanczos solver

The panels are 26 Balding-Nichols populations (the population count of the 1000 Genomes panel) with
population Fst of 0.02 to 0.12 and ancestral frequencies of 0.05 to 0.5. The products of the mixed
and FP32 precisions carry 21 to 24 bits, so the programs keep U, S and V as 32-bit values;
frequencies, covariances, 64-bit r2 and 64-bit products stay as they are.
"""
import math

import numpy as np
import torch

import pcaone_b200 as pb

POPS = 26


# ------------------------------------------------------------------ cases
def listed():
    return [
        # a small study: a few hundred samples, one call from records to PCs (latency, launches)
        dict(name="pca-small-whole", kind="pca", how="whole", n=203, m=1500, k=4, svd=1, bands=64, maxp=20,
             tol=1e-4, precision="mixed", miss=0.02),
        # Halko with a fixed number of power iterations, the package's smallest benchmark
        dict(name="halko-2000x50000", kind="pca", how="resident", n=2000, m=50000, k=10, svd=1, bands=64, maxp=7,
             tol=0.0, precision="mixed", miss=0.01),
        # an ordinary cohort with odd sizes, default flags, everything from the records on
        dict(name="winsvd-5003x80021-whole", kind="pca", how="whole", n=5003, m=80021, k=10, svd=2, bands=64,
             maxp=20, tol=1e-4, precision="mixed", miss=0.01),
        # the largest: a biobank-sized panel, twenty PCs, default flags
        dict(name="winsvd-20000x500000", kind="pca", how="resident", n=20000, m=500000, k=20, svd=2, bands=64,
             maxp=20, tol=1e-4, precision="mixed", miss=0.005),
        # the binding's default precision on a pruned SNP set
        dict(name="winsvd-fp32-1502x30011", kind="pca", how="resident", n=1502, m=30011, k=5, svd=2, bands=64,
             maxp=20, tol=1e-4, precision="fp32", miss=0.02),
        # out of core: records in host memory, windows copied to two device slots in every epoch
        dict(name="winsvd-8001x120000-streamed", kind="pca", how="streamed", n=8001, m=120000, k=10, svd=2, bands=64,
             maxp=20, tol=1e-4, precision="mixed", miss=0.01, slot_mb=128),
        # low-coverage or array data with a tenth of the entries missing
        dict(name="emu-5000x100000", kind="emu", n=5000, m=100000, k=10, bands=64, maxp=20, tol=1e-4),
        # low-depth sequencing
        dict(name="pcangsd-2001x60000", kind="pcangsd", n=2001, m=60000, k=6, bands=64, maxp=20, tol=1e-4),
        dict(name="grm-1501x40000", kind="grm", n=1501, m=40000, k=6),
        # LD of a chromosome arm, adjusted for population structure
        dict(name="ld-5000x60000-adjusted", kind="ld", n=5000, m=60000, k=10, bp=1000000, f64=False, miss=0.01),
        # the pairs a clumping or pruning pass compares, on one region
        dict(name="ld-2504x5000-f64", kind="ld", n=2504, m=5000, k=0, bp=250000, f64=True, miss=0.01),
        # one operator call of the Lanczos solver (64-bit products, one vector)
        dict(name="gram-3000x60001-fp64", kind="gram", n=3000, m=60001, cols=1, precision="fp64", miss=0.01),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pca", "pca", "pca", "pca", "emu", "pcangsd", "grm", "ld", "gram"])
    if kind == "pca":
        how = rng.choice(["resident", "resident", "whole", "streamed"])
        precision = "mixed" if how == "streamed" else rng.choice(["mixed", "mixed", "mixed", "fp32"])
        n = _log(rng, 200, 20000)
        m = _log(rng, 5000, min(500000, (2e9 if precision == "mixed" else 3e8) / n))
        svd = rng.choice([1, 2, 2])
        return dict(kind="pca", how=how, n=n, m=m, k=rng.randint(2, 20 if n >= 1000 else 5), svd=svd,
                    bands=rng.choice([16, 64]), maxp=rng.choice([7, 20]), tol=rng.choice([0.0, 1e-4]) if svd == 1 else 1e-4,
                    precision=precision, miss=rng.choice([0.0, 0.005, 0.02]),
                    **({"slot_mb": rng.choice([32, 128])} if how == "streamed" else {}))
    if kind == "emu":
        n = _log(rng, 500, 10000)
        return dict(kind="emu", n=n, m=_log(rng, 10000, min(200000, 4e8 / n)), k=rng.randint(4, 12), bands=64, maxp=20,
                    tol=1e-4)
    if kind == "pcangsd":
        n = _log(rng, 100, 4000)
        return dict(kind="pcangsd", n=n, m=_log(rng, 10000, min(200000, 1.5e8 / n)), k=rng.randint(2, 8), bands=64,
                    maxp=20, tol=1e-4)
    if kind == "grm":
        n = _log(rng, 100, 3000)
        return dict(kind="grm", n=n, m=_log(rng, 5000, min(100000, 1e8 / n)), k=rng.randint(2, 8))
    if kind == "ld":
        n = _log(rng, 200, 10000)
        return dict(kind="ld", n=n, m=_log(rng, 2000, min(60000, 4e8 / n)), k=rng.choice([0, 3, 10]),
                    bp=rng.choice([100000, 250000, 1000000]), f64=rng.random() < 0.3, miss=rng.choice([0.0, 0.02]))
    n = _log(rng, 200, 10000)
    return dict(kind="gram", n=n, m=_log(rng, 5000, min(300000, 5e8 / n)), cols=rng.choice([1, 1, 5, 20]),
                precision="fp64", miss=rng.choice([0.0, 0.02]))


# ------------------------------------------------------------------ inputs
def _frequencies(n, m, gen):
    """Population of each sample, and each SNP's allele frequency in each population."""
    dev = gen.device
    pop = torch.randint(0, POPS, (n,), generator=gen, device=dev)
    fst = torch.linspace(0.02, 0.12, POPS, device=dev)
    anc = 0.05 + 0.45 * torch.rand(m, 1, generator=gen, device=dev)
    z = torch.randn(m, POPS, generator=gen, device=dev)
    return pop, (anc + (fst * anc * (1 - anc)).sqrt() * z).clamp_(0.02, 0.98)


def _rows(n):
    return max(1, (1 << 26) // n)


def _records(case, seed, missing=None):
    """PLINK records (m x ceil(n/4) bytes, on the GPU): Hardy-Weinberg genotypes, entries missing at
    random with rate case["miss"] or the per-sample rates `missing`."""
    n, m = case["n"], case["m"]
    gen = torch.Generator("cuda").manual_seed(int(seed))
    pop, freq = _frequencies(n, m, gen)
    miss = torch.full((n,), float(case.get("miss", 0.0)), device="cuda") if missing is None else missing
    n4 = (n + 3) // 4
    out = torch.empty(m, n4, dtype=torch.uint8, device="cuda")
    for a in range(0, m, _rows(n)):
        p = freq[a:a + _rows(n)][:, pop]
        u = torch.rand(p.shape, generator=gen, device="cuda")
        q = 1 - p
        v = (u - miss) / (1 - miss)
        # A1 copies 0, 1, 2 are codes 3, 2, 0; missing is code 1
        code = torch.where(v < q * q, 3, torch.where(v < 1 - p * p, 2, 0)).to(torch.uint8)
        code[u < miss] = 1
        code = torch.nn.functional.pad(code, (0, 4 * n4 - n)).view(-1, n4, 4)
        out[a:a + p.shape[0]] = code[:, :, 0] | code[:, :, 1] << 2 | code[:, :, 2] << 4 | code[:, :, 3] << 6
    return out


def _missing_rates(case, seed):
    """Per-sample missing rates, Beta(2, 18)."""
    r = np.random.default_rng(int(seed)).beta(2, 18, case["n"]).astype(np.float32)
    return torch.from_numpy(r).cuda()


def _likelihoods(case, seed):
    """Genotype likelihood pairs (m x 2n FP32, on the GPU) from reads of depth Poisson(4) with error
    rate 0.01."""
    n, m = case["n"], case["m"]
    gen = torch.Generator("cuda").manual_seed(int(seed))
    pop, freq = _frequencies(n, m, gen)
    out = torch.empty(m, n, 2, device="cuda")
    rate = torch.tensor([0.01, 0.5, 0.99], device="cuda")
    for a in range(0, m, _rows(4 * n)):
        p = freq[a:a + _rows(4 * n)][:, pop]
        u = torch.rand(p.shape, generator=gen, device="cuda")
        q = 1 - p
        g = (u > q * q).long() + (u > 1 - p * p)
        depth = torch.poisson(torch.full_like(p, 4.0), generator=gen)
        alt = torch.binomial(depth, rate[g], generator=gen)
        like = torch.stack([alt * r.log() + (depth - alt) * (1 - r).log() for r in rate]).softmax(0)
        out[a:a + p.shape[0], :, 0], out[a:a + p.shape[0], :, 1] = like[0], like[1]
    return out.view(m, 2 * n)


def _factors(case, seed):
    """U (n x k, orthonormal), S and V (m x k) such as a PCA of the matrix gives."""
    n, m, k = case["n"], case["m"], case["k"]
    rng = np.random.default_rng(int(seed) + 1)
    U = np.linalg.qr(rng.standard_normal((n, k)))[0]
    V = rng.standard_normal((m, k)) / math.sqrt(m)
    S = 0.05 * math.sqrt(n * m) * np.linspace(1.0, 0.3, k)
    return np.asfortranarray(U), S, np.asfortranarray(V)


def _shuffle(case, seed):
    """SNP order of an in-core shuffle."""
    return np.random.default_rng(int(seed) + 3).permutation(case["m"]).astype(np.int32)


def _windows(case):
    """Windows of the SNPs within bp of each lead SNP, one SNP per kilobase on average: one array's
    map, the same for every panel."""
    step = np.random.default_rng(2).integers(1, 2000, case["m"])
    return pb.ld_windows(np.cumsum(step), [case["m"] - 1], case["bp"])


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    s = dict(case=case, ctx=pb.GpuContext(0))
    ctx = s["ctx"]
    if kind in ("pcangsd", "grm"):
        P = _likelihoods(case, seed).cpu().numpy().T
        ctx.load_gl(P)
        if kind == "grm":
            ctx.gl_freq()
            s["factors"] = _factors(case, seed)
        return s
    packed = _records(case, seed, _missing_rates(case, seed) if kind == "emu" else None).cpu().numpy()
    if kind == "pca" and case["svd"] == 2:
        s["perm"] = _shuffle(case, seed)
    if case.get("how") == "whole":
        s["packed"] = packed
        return s
    if case.get("how") == "streamed":
        ctx.load_bed_host(packed, n, slot_bytes=case["slot_mb"] << 20)
    else:
        ctx.load_bed(packed, n)
    if kind == "emu":
        ctx.permute(_shuffle(case, seed))
    elif "perm" in s:
        ctx.permute(s["perm"])
    if kind == "ld":
        s["ws"], s["we"] = _windows(case)
        s["U"] = _factors(case, seed)[0] if case["k"] else None
    if kind == "gram":
        s["X"] = np.asfortranarray(np.random.default_rng(int(seed)).standard_normal((n, case["cols"])))
    return s


# ------------------------------------------------------------------ one pass
def _keep(U, S, V):
    return dict(U=torch.from_numpy(U).float(), S=torch.from_numpy(S).float(), V=torch.from_numpy(V).float())


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "pca":
        if case["how"] == "whole":
            ctx.load_bed(state["packed"], case["n"])
            if "perm" in state:
                ctx.permute(state["perm"])
        r = ctx.rsvd(k=case["k"], svd=case["svd"], bands=case["bands"], maxp=case["maxp"], tol=case["tol"],
                     precision=case["precision"])
        return _keep(r.U, r.S, r.V)
    if kind == "emu":
        _, S, U, V, _, _ = pb.emu_loop(ctx, k=case["k"], bands=case["bands"], maxp=case["maxp"], tol=case["tol"],
                                       maxiter=1)
        return _keep(U, S, V)
    if kind == "pcangsd":
        kw = dict(k=case["k"], svd=2, bands=case["bands"], maxp=case["maxp"], tol=case["tol"],
                  precision="fp32", standardize=False)
        F, _ = ctx.gl_freq()
        ctx.gl_update()
        r = ctx.rsvd(carry=False, **kw)
        ctx.gl_update(r.U, r.S, r.V)
        r = ctx.rsvd(carry=True, **kw)
        return dict(F=F, **_keep(r.U, r.S, r.V))
    if kind == "grm":
        return ctx.gl_grm(*state["factors"], vectors=False)[0]
    if kind == "ld":
        return ctx.ld_r2(state["ws"], state["we"], state["U"], f64=case["f64"])
    return ctx.gram_product(state["X"], precision=case["precision"])


def _width(case):
    return case["k"] + max(10, case["k"])


def _epochs(case):
    """Epochs a PCA cannot do without: all of them with tol 0, else two (Halko) or those in which
    the windows grow to the whole matrix."""
    if case.get("svd", 2) == 1:
        return case["maxp"] + 1 if case["tol"] == 0 else 2
    return int(math.log2(case["bands"])) + 1


def work(case):
    n, m, kind = case["n"], case["m"], case["kind"]
    if kind == "pca":
        return dict(bytes=n * m / 4 + 4 * (n + m) * case["k"], flops=4.0 * n * m * _width(case) * _epochs(case))
    if kind == "emu":
        return dict(bytes=n * m / 4 + 4 * (n + m) * case["k"], flops=3 * 4.0 * n * m * _width(case) * _epochs(case))
    if kind == "pcangsd":
        return dict(bytes=16.0 * n * m + 4 * (n + m) * case["k"], flops=2 * 4.0 * n * m * _width(case) * _epochs(case))
    if kind == "grm":
        return dict(bytes=16.0 * n * m + 8.0 * n * n, flops=1.0 * n * n * m)
    if kind == "ld":
        pairs = m * min(case["bp"] / 1000.0, m / 2)
        return dict(bytes=n * m / 4 + (8 if case["f64"] else 4) * pairs, flops=8.0 * n * pairs)
    return dict(bytes=n * m / 4 + 16.0 * n * case["cols"], flops=4.0 * n * m * case["cols"])


# ------------------------------------------------------------------ the same in 64 bits
def _omega(n, l, seed=101):
    """libstdc++'s normal_distribution on a default_random_engine (minstd_rand0), column-major."""
    p = 2147483647
    draws = 4 * (int(n * l / 1.5) + 2000)
    x = np.array([16807 * seed % p], dtype=np.int64)
    while len(x) < draws:
        x = np.concatenate([x, x * pow(16807, len(x), p) % p])
    g, r = x[:draws].astype(np.float64) - 1, float(p - 1)
    u = 2 * ((g[0::2] + g[1::2] * r) / (r * r)) - 1
    a, b = u[0::2], u[1::2]
    r2 = a * a + b * b
    ok = (r2 <= 1) & (r2 > 0)
    a, b, r2 = a[ok], b[ok], r2[ok]
    f = np.sqrt(-2 * np.log(r2) / r2)
    z = np.stack([b * f, a * f], 1).reshape(-1)[:n * l]
    return torch.from_numpy(z.reshape(l, n).T.copy()).cuda()


class _Rsvd64:
    """Randomised SVD of Z^T (m x n, 64 bits): Halko or window-based power iterations on the seeded
    sketch; successive calls of the window-based form carry its window sums on."""

    def __init__(self, n, l, case):
        self.h = [torch.zeros(n, l, dtype=torch.float64, device="cuda") for _ in range(2)]
        self.omega0, self.case = _omega(n, l), case

    def orth(self, H, last):
        Q = torch.linalg.qr(H)[0]
        flip = (last - Q).abs().sum(0) > 2 * (last + Q).abs().sum(0)
        return torch.where(flip, -Q, Q)

    def __call__(self, Zt):
        c, m = self.case, Zt.shape[0]
        k, p, bands = c["k"], c["maxp"], c["bands"]
        O, before = self.omega0, None
        G = torch.empty(m, O.shape[1], dtype=torch.float64, device="cuda")
        bs, band, pi = -(-m // bands), 1, 0
        while pi <= p:
            if c.get("svd", 2) == 1:
                if pi:
                    O = self.orth(H, O)
                G = Zt @ O
                H = Zt.T @ G
            else:
                if 2 ** pi >= bands:
                    self.h = [torch.zeros_like(h) for h in self.h]
                band, i = min(2 * band, bands), 1
                for b in range(bands):
                    w = slice(b * bs, min(m, (b + 1) * bs))
                    G[w] = Zt[w] @ O
                    t = 0 if i <= band // 2 else 1
                    self.h[t] = self.h[t] + Zt[w].T @ G[w]
                    near = pi > 0 and b + 1 == 2 ** (pi - 1) and 2 ** pi < bands
                    if (b + 1 >= band or near) and (i in (band, band // 2) or near):
                        H = self.h[0] + self.h[1]
                        O = self.orth(H, O)
                        self.h[0 if i == band else 1] = torch.zeros_like(H)
                        if i == band:
                            i = 0
                    i += 1
            Q, R = torch.linalg.qr(G)
            U, S, Vh = torch.linalg.svd(torch.linalg.solve_triangular(R.T, H.T, upper=False), full_matrices=False)
            now = Vh.T[:, :k]
            if pi:
                diff = 1 - (now.T @ before).norm(dim=0).mean().item()
                if diff < c["tol"] or pi == p:
                    if c.get("svd", 2) == 2 and 2 ** pi < bands:
                        p = int(math.log2(bands))
                        pi += 1
                        continue
                    break
            before, pi = now, pi + 1
        return now, S[:k], Q @ U[:, :k]


def _dense(case, seed):
    """Centred genotypes (m x n, 64 bits, missing 0), allele frequencies and the missing mask."""
    n = case["n"]
    packed = _records(case, seed, _missing_rates(case, seed) if case["kind"] == "emu" else None)
    if case["kind"] == "emu" or case.get("svd") == 2:
        packed = packed[torch.from_numpy(_shuffle(case, seed).astype(np.int64)).cuda()]
    code = torch.stack([packed >> s & 3 for s in (0, 2, 4, 6)], 2).view(packed.shape[0], -1)[:, :n]
    x = torch.tensor([1.0, 0.0, 0.5, 0.0], dtype=torch.float64, device="cuda")[code.int()]
    miss = code == 1
    F = x.sum(1) / (n - miss.sum(1))
    return torch.where(miss, 0.0, x - F[:, None]), F, miss


def _scale(F):
    return 1 / (2 * F * (1 - F)).sqrt()


def _posterior(P, F, pt):
    p0 = P[:, 0::2] * (1 - pt) ** 2
    p1 = P[:, 1::2] * 2 * pt * (1 - pt)
    p2 = (1 - P[:, 0::2] - P[:, 1::2]) * pt ** 2
    t = p0 + p1 + p2
    return p0 / t, p1 / t, p2 / t


def _gl_freq64(P):
    F = torch.full((P.shape[0],), 0.25, dtype=torch.float64, device="cuda")
    for _ in range(100):
        _, p1, p2 = _posterior(P, F, F[:, None])
        new = (p1 + 2 * p2).sum(1) / P.shape[1]
        done = (new - F).square().mean().sqrt() < 1e-6
        F = new
        if done:
            break
    return F


def exact(case, seed):
    kind, n, m = case["kind"], case["n"], case["m"]
    if n * m > 1e9:
        return None
    if kind == "pca":
        Z, F, _ = _dense(case, seed)
        S = _Rsvd64(n, _width(case), case)(Z * _scale(F)[:, None])[1]
        return dict(U=None, S=S.cpu(), V=None)
    if kind == "emu":
        return _emu64(case, seed)
    if kind in ("pcangsd", "grm"):
        P = _likelihoods(case, seed).double()
        F = _gl_freq64(P)
        f = F[:, None]
        if kind == "grm":
            U, S, V = (torch.from_numpy(x).cuda() for x in _factors(case, seed))
            p0, p1, p2 = _posterior(P, F, ((V * S) @ U.T / 2 + f).clamp(1e-4, 1 - 1e-4))
            E = (p1 + 2 * p2 - 2 * f) * _scale(F)[:, None]
            d = (4 * f * f * p0 + (1 - 2 * f) ** 2 * p1 + (2 - 2 * f) ** 2 * p2) / (2 * f * (1 - f))
            C = E.T @ E
            C.diagonal().copy_(d.sum(0))
            return (C / m).cpu()
        rsvd = _Rsvd64(n, _width(case), case)
        U, S, V = rsvd(_mean(P, F, f))
        U, S, V = rsvd(_mean(P, F, ((V * S) @ U.T / 2 + f).clamp(1e-4, 1 - 1e-4)))
        return dict(F=F.cpu(), U=None, S=S.cpu(), V=None)
    if kind == "ld":
        G, _, _ = _dense(case, seed)
        if case["k"]:
            U = torch.from_numpy(_factors(case, seed)[0]).cuda()
            G -= (G @ U) @ U.T
        G /= G.norm(dim=1, keepdim=True)
        ws, we = _windows(case)
        out, reach = [], int(we.max())
        for a in range(0, len(ws), 512):
            w, e = torch.from_numpy(ws[a:a + 512]).cuda(), torch.from_numpy(we[a:a + 512]).cuda()
            lo = int(w[0])
            hi = min(m, lo + 512 + reach)
            at = torch.arange(lo, hi, device="cuda")
            inside = (at > w[:, None]) & (at < (w + e)[:, None])
            out.append((G[w] @ G[lo:hi].T).square()[inside])
        return torch.cat(out).cpu()
    Z, F, _ = _dense(case, seed)
    Z *= _scale(F)[:, None]
    X = torch.from_numpy(np.random.default_rng(int(seed)).standard_normal((n, case["cols"]))).cuda()
    return (Z.T @ (Z @ X)).cpu()


def _mean(P, F, pt):
    _, p1, p2 = _posterior(P, F, pt)
    return p1 + 2 * p2 - 2 * F[:, None]


def _emu64(case, seed):
    Z, F, miss = _dense(case, seed)
    # after the in-core shuffle the reference clips and standardises SNP j with the frequency of
    # the SNP that was at position j of the input
    Fl = torch.empty_like(F)
    Fl[torch.from_numpy(_shuffle(case, seed).astype(np.int64)).cuda()] = F
    Fl = Fl[:, None]
    rsvd = _Rsvd64(case["n"], _width(case), case)
    U, S, V = rsvd(Z)
    for last in (False, True):
        Z = torch.where(miss, torch.minimum(torch.maximum((V * S) @ U.T, -Fl), 1 - Fl), Z)
        U, S, V = rsvd(Z * _scale(Fl) if last else Z)
    return dict(U=None, S=S.cpu(), V=None)
