"""The work whose speed is followed: calls of the package's public entry points at the
sizes of the benchmark's configurations and around them, from the smallest calls to a
single-step problem of 200,000 animals.

Each kind of case is one step of a genetic evaluation, in the order a program runs them:
``grm`` (BED bytes to G), ``ginv`` (G to its eigen-bent inverse), ``hinv`` (pedigree and G
to the single-step H^-1 blocks), ``solve`` (one MME solve), ``dense`` (AI-REML of a small
data set, dense exact steps), ``em`` / ``ssem`` (EM-REML of a large one, GBLUP and
single-step), ``final`` (final single-step solve with standard errors), ``snp`` (genotype
products), ``batch`` (many small problems at once), ``mt`` (multi-trait).

Solves run to relative residuals of 1e-12 or 1e-13, at which breeding values are settled
to 1e-8 (the parity bar of this package's tests); at 1e-10 they are not.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import cosmicblup_gb300 as cb
from cosmicblup_gb300._lib import ptr
from cosmicblup_gb300.mme import FP64, MIXED
from cosmicblup_gb300.synth import simulate_pedigree
from cosmicblup_gb300.vce import MODE_AUTO, MODE_EM

MAGIC = np.array([0x6C, 0x1B, 0x01], dtype=np.uint8)
MIN_MAF = 0.01
START = (0.5, 0.5)           # starting variances, as in the benchmark


def listed():
    return [
        # the smallest GRM of the batched configuration: launches and copies count
        {"name": "grm_n501", "kind": "grm", "n": 501, "m": 5003, "counts": True},
        # a national-evaluation GRM of a 50k chip, G read back by the program
        {"name": "grm_n12000", "kind": "grm", "n": 12000, "m": 40001, "counts": False},
        # G^-1 of a mid-size genotyped population, left on the device and read back
        {"name": "ginv_n5003", "kind": "ginv", "n": 5003, "m": 20000, "ridge": 0.0},
        # single-step set-up: A22, tuneG, blend, both inverses
        {"name": "hinv_3000_of_15000", "kind": "hinv", "gens": 10, "per": 1500, "gen_g": 2, "m": 9000},
        # one breeding-value solve of a small herd, FP64: latency
        {"name": "solve_n503_fp64", "kind": "solve", "n": 503, "m": 5003, "nrhs": 1, "mixed": False},
        # the plain GBLUP configuration, AI-REML to convergence
        {"name": "dense_n2000", "kind": "dense", "n": 2000, "m": 10000, "levels": 2},
        # the large GBLUP configuration: three EM-REML iterations, 32 or more probes
        {"name": "em_n20000", "kind": "em", "n": 20000, "m": 50000, "levels": 200},
        # the single-step configuration: three EM-REML iterations, each with its gradient
        {"name": "ssem_200000_20000", "kind": "ssem", "gens": 10, "per": 20000, "gen_g": 1, "m": 50000, "levels": 500,
         "probes": 64},
        # final single-step solve with fixed-effect standard errors, FP64 (the default precision)
        {"name": "final_se_15000_3000", "kind": "final", "gens": 10, "per": 1500, "gen_g": 2, "m": 9000, "levels": 33,
         "mixed": False},
        # Z'v and Z w on a 50k chip, one vector: one iteration of a matrix-free solver
        {"name": "snp_n20000_m50000", "kind": "snp", "n": 20000, "m": 50000, "nvec": 1},
        # a batch of uneven small problems on one worker, BED to variance components
        {"name": "batch_8", "kind": "batch", "nprob": 8, "n_lo": 500, "n_hi": 2500, "m": 5000},
        # three traits on one small population: variance components and breeding values
        {"name": "mt_n1003_t3", "kind": "mt", "n": 1003, "m": 5003, "traits": 3},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["grm", "ginv", "hinv", "solve", "dense", "em", "ssem", "final", "snp", "batch", "mt"])
    c = {"kind": kind}
    if kind == "grm":
        c.update(n=_log(rng, 300, 12000), m=_log(rng, 3000, 40000), counts=rng.random() < 0.25)
    elif kind == "ginv":
        c.update(n=_log(rng, 400, 5000), m=_log(rng, 6500, 20000), ridge=rng.choice([0.0, 0.0, 0.01]))
    elif kind == "hinv":
        per = _log(rng, 150, 1500)
        c.update(gens=rng.randint(3, 10), per=per, gen_g=rng.randint(1, 2), m=4 * per + rng.randint(500, 2500))
    elif kind == "solve":
        c.update(n=_log(rng, 400, 6000), m=_log(rng, 8000, 20000), nrhs=_log(rng, 1, 40), mixed=rng.random() < 0.5)
    elif kind == "dense":
        c.update(n=_log(rng, 300, 2000), m=_log(rng, 4000, 10000), levels=rng.randint(2, 12))
    elif kind == "em":
        n = _log(rng, 5100, 20000)
        c.update(n=n, m=int(2.5 * n), levels=rng.randint(2, 200))
    elif kind == "ssem":
        per = _log(rng, 600, 20000)
        c.update(gens=rng.randint(5, 10), per=per, gen_g=1, m=max(2000, int(2.5 * per)), levels=rng.randint(20, 500),
                 probes=rng.choice([16, 32, 64]))
    elif kind == "final":
        per = _log(rng, 150, 1500)
        c.update(gens=rng.randint(4, 10), per=per, gen_g=rng.randint(1, 2), m=4 * per + rng.randint(500, 2500),
                 levels=rng.randint(2, 33), mixed=rng.random() < 0.5)
    elif kind == "snp":
        n = _log(rng, 500, 20000)
        c.update(n=n, m=_log(rng, 5000, 50000), nvec=_log(rng, 1, 12) if n < 8000 else 1)
    elif kind == "batch":
        c.update(nprob=rng.randint(3, 8), n_lo=500, n_hi=rng.randint(900, 2500), m=rng.randint(5000, 9000))
    else:
        c.update(n=_log(rng, 300, 1003), m=rng.randint(4000, 6000), traits=rng.randint(2, 3))
    return c


# ---- inputs ----------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(1_000_003 * int(seed) + 17)


def _calls(g, n, m, miss=0.02):
    """Genotype calls (m x n, copies of allele 1, -1 = missing) in Hardy-Weinberg
    proportions, frequencies U(0.01, 0.5), in blocks of SNPs."""
    p = torch.rand(m, generator=g, device="cuda") * 0.49 + 0.01
    for j in range(0, m, 4096):
        q = p[j:j + 4096, None]
        u = torch.rand(q.shape[0], n, generator=g, device="cuda")
        x = (u < q * q).to(torch.int8) + (u < q * (2 - q)).to(torch.int8)
        x[torch.rand(x.shape, generator=g, device="cuda") < miss] = -1
        yield j, x


def _pack(x):
    """PLINK codes of a block of calls, four samples a byte."""
    code = torch.tensor([3, 2, 0, 1], dtype=torch.uint8, device="cuda")[x.long() % 4]
    k, n = x.shape
    pad = torch.zeros(k, -n % 4, dtype=torch.uint8, device="cuda")
    c = torch.cat([code, pad], 1).view(k, -1, 4)
    return c[:, :, 0] | (c[:, :, 1] << 2) | (c[:, :, 2] << 4) | (c[:, :, 3] << 6)


def _bed(blocks):
    return np.concatenate([MAGIC] + [_pack(x).cpu().numpy().reshape(-1) for _, x in blocks])


def _centre(x, dtype):
    """Centred genotypes of a block (missing = 0) and 2pq; means are floats as the package keeps them."""
    ok = x >= 0
    f = torch.where(ok, x, 0).sum(1, dtype=torch.float64) / (2.0 * ok.sum(1).clamp(min=1))
    keep = torch.minimum(f, 1 - f) >= float(np.float32(MIN_MAF))
    z = torch.where(ok, x.to(dtype) - (2 * f).float().to(dtype)[:, None], 0.0) * keep[:, None]
    return z, (2 * f * (1 - f)).float().double() * keep, f, keep


def _vanraden(blocks, n, dtype):
    """G = Z Z' / sum 2pq.  float32 products run as TF32 (an input matrix is rounded once more, that is all)."""
    G = torch.zeros(n, n, dtype=dtype, device="cuda")
    s, old = 0.0, torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = True
    for _, x in blocks:
        z, w, _, _ = _centre(x, dtype)
        G.addmm_(z.T, z)
        s += float(w.sum())
    torch.backends.cuda.matmul.allow_tf32 = old
    return G.div_(s)


def _pinned(shape, dtype=torch.float64):
    """A page-locked host array, as a program that reuses its buffers holds them."""
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


def _host(t):
    a = _pinned(tuple(t.shape))
    torch.from_numpy(a).copy_(t)
    return a


def _records(rng, u, levels):
    """One record an animal: mean, class effect, breeding value and residual; the design as CSR."""
    n = u.size
    lvl = rng.integers(0, levels, size=n)
    y = 10.0 + rng.normal(size=levels)[lvl] + u + rng.normal(0.0, math.sqrt(0.6), size=n)
    two = lvl > 0
    fp = np.zeros(n + 1, dtype=np.int64)
    np.cumsum(1 + two, out=fp[1:])
    fc = np.zeros(fp[-1], dtype=np.int32)
    fc[fp[:-1][two] + 1] = lvl[two]
    return y, np.arange(1, n + 1, dtype=np.int32), (fp, fc, np.ones(fp[-1])), levels


def _bent_inverse32(G):
    """Inverse of a centred G whose null direction (all ones) is bent to 1e-6, made in float32: an input."""
    n = G.shape[0]
    G = G.float() + 1.0 / n
    X = torch.cholesky_inverse(torch.linalg.cholesky(G)).double()
    X = 0.5 * (X + X.T)
    s = X.sum(0) / n
    X -= s[:, None] + s[None, :] - s.sum() / n
    return X.add_(1e6 / n)


def _pedigree(case, seed):
    """Discrete generations, founders first; the last gen_g of them are genotyped.  Returns (sire, dam)."""
    gens, per = case["gens"], case["per"]
    sire, dam = simulate_pedigree(gens, per, max(2, per // 40), per // 2, seed=9 * seed + 5)
    return sire, dam


def _relationships(case, sire, dam, seed, dtype):
    """A^-1 (CSR), A22, G and the genotyped rows: A by generations, genotypes by gene dropping."""
    gens, per, k = case["gens"], case["per"], case["gen_g"]
    q, m = gens * per, case["m"]
    g = _gen(seed + 77)
    ps = torch.from_numpy(sire).cuda().view(gens, per)
    pd = torch.from_numpy(dam).cuda().view(gens, per)
    # relationships: A of one generation from the one before it
    A = torch.eye(per, dtype=dtype, device="cuda")
    d = [torch.ones(per, dtype=torch.float64, device="cuda")]
    blocks = {0: A}
    for t in range(1, gens):
        s, e = ps[t] - (t - 1) * per, pd[t] - (t - 1) * per
        ws, we = (ps[t] >= 0).to(dtype) * 0.5, (pd[t] >= 0).to(dtype) * 0.5
        s, e = s.clamp(min=0), e.clamp(min=0)
        cross = A[s] * ws[:, None] + A[e] * we[:, None]          # A(t, t - 1)
        F = 0.5 * A[s, e] * (ws * we * 4)
        A = cross[:, s] * ws[None, :] + cross[:, e] * we[None, :]
        d.append((1 + F - A.diagonal()).double())
        A.diagonal().copy_(1 + F)
        blocks = {0: blocks.get(1, A), 1: A, 2: cross} if t == gens - 1 else {1: A}
    A22 = A if k == 1 else torch.cat([torch.cat([blocks[0], blocks[2].T], 1), torch.cat([blocks[2], A], 1)], 0)
    # A^-1 by Henderson's rules: d_i^-1 (1, -1/2, -1/2)' (1, -1/2, -1/2)
    di = 1.0 / torch.cat(d)
    i = torch.arange(q, device="cuda")
    par = [(i, torch.ones(q, dtype=torch.float64, device="cuda")), (ps.reshape(-1), None), (pd.reshape(-1), None)]
    par = [(x, torch.where(x >= 0, -0.5, 0.0).double() if w is None else w) for x, w in par]
    key = torch.cat([(x.clamp(min=0) * q + y.clamp(min=0)) for x, _ in par for y, _ in par])
    val = torch.cat([a * b * di for _, a in par for _, b in par])
    ok = val != 0
    key, pos = torch.unique(key[ok], return_inverse=True)
    val = torch.zeros(key.numel(), dtype=torch.float64, device="cuda").index_put_((pos,), val[ok], accumulate=True)
    row = torch.div(key, q, rounding_mode="floor")
    aptr = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), torch.bincount(row, minlength=q).cumsum(0)])
    # G: haplotypes dropped through the pedigree, in blocks of SNPs
    G = torch.zeros(k * per, k * per, dtype=dtype, device="cuda")
    tot = 0.0
    old, torch.backends.cuda.matmul.allow_tf32 = torch.backends.cuda.matmul.allow_tf32, True
    for j in range(0, m, 5000):
        w = min(5000, m - j)
        p = torch.rand(w, generator=g, device="cuda") * 0.49 + 0.01

        def fresh():
            return torch.rand(per, w, generator=g, device="cuda") < p
        hap = (fresh(), fresh())
        x = [hap[0].to(torch.int8) + hap[1].to(torch.int8)]
        for t in range(1, gens):
            new = []
            for par_t in (ps[t], pd[t]):
                idx = (par_t - (t - 1) * per).clamp(min=0)
                pick = torch.randint(0, 2, (per, w), generator=g, device="cuda", dtype=torch.uint8).bool()
                h = torch.where(pick, hap[0][idx], hap[1][idx])
                new.append(torch.where((par_t >= 0)[:, None], h, fresh()))
            hap = tuple(new)
            if t >= gens - k:
                x.append(hap[0].to(torch.int8) + hap[1].to(torch.int8))
        z, tq, _, _ = _centre(torch.cat(x[-k:]).T.contiguous(), dtype)
        G.addmm_(z.T, z)
        tot += float(tq.sum())
    torch.backends.cuda.matmul.allow_tf32 = old
    G.div_(tot)
    gmap = np.arange(q - k * per, q, dtype=np.int32)
    csr = (aptr.cpu().numpy(), (key % q).to(torch.int32).cpu().numpy(), val.cpu().numpy())
    return csr, A22, 0.5 * (G + G.T), gmap


def _tune(G, A):
    """G scaled and shifted to the means of A's diagonal and off-diagonal."""
    n = G.shape[0]
    gd, ad = G.diagonal().sum() / n, A.diagonal().sum() / n
    go, ao = (G.sum() - gd * n) / (n * (n - 1.0)), (A.sum() - ad * n) / (n * (n - 1.0))
    b = (ad - ao) / (gd - go)
    return G * b + (ad - b * gd)


def _ped_values(rng, sire, dam, per):
    a = rng.normal(size=sire.size)
    for t in range(per, sire.size, per):
        s, e = sire[t:t + per], dam[t:t + per]
        a[t:t + per] = (0.5 * np.where(s >= 0, a[s], 0) + 0.5 * np.where(e >= 0, a[e], 0)
                        + a[t:t + per] * math.sqrt(0.5))
    return a * math.sqrt(0.35)


def _inv32(A):
    X = torch.cholesky_inverse(torch.linalg.cholesky(A.float()))
    return 0.5 * (X + X.T)


def _grm_call(h, bed, n, m, G=None, xx=None, freqs=None):
    s, k = C.c_double(0.0), C.c_int64(0)
    h.check(cb.lib().cbx_grm_bed(h.raw, ptr(bed), bed.size, n, m, C.c_float(MIN_MAF), 1, 2048, ptr(G), ptr(xx),
                                 ptr(freqs), C.byref(s), C.byref(k)))
    return s.value, k.value


def _phenotypes(case, seed, t):
    """Records of a GBLUP data set and its G in the given type."""
    n = case["n"]
    G = _vanraden(_calls(_gen(seed), n, case["m"], 0.0), n, t)
    rng = np.random.default_rng(seed + 31)
    w = torch.from_numpy(rng.normal(size=n)).to("cuda", t)
    # a draw with covariance close to 0.4 G (one Newton-Schulz step towards its square root is enough here)
    g = (0.75 * (G @ w) + 0.25 * w).double().cpu().numpy() * math.sqrt(0.4)
    return G, _records(rng, g, case.get("levels", 2))


def _mt_data(case, seed, G):
    n, t = case["n"], case["traits"]
    rng = np.random.default_rng(seed + 41)
    L = np.linalg.cholesky(np.array([[0.4, 0.2, -0.1], [0.2, 0.5, 0.1], [-0.1, 0.1, 0.5]])[:t, :t])
    z = (G @ torch.from_numpy(rng.normal(size=(n, t))).cuda()).cpu().numpy()
    X = np.stack([np.ones(n), rng.integers(0, 2, n).astype(float)], 1)
    return 10.0 + X @ rng.normal(size=(2, t)) + z @ L.T + rng.normal(size=(n, t)) * 0.75, X


def prepare(case, seed):
    kind = case["kind"]
    h = cb.Handle(0)
    s = {"case": case, "h": h}
    rng = np.random.default_rng(seed + 21)
    if kind in ("grm", "ginv", "snp"):
        n, m = case["n"], case["m"]
        bed = _bed(_calls(_gen(seed), n, m))
        if kind == "grm":
            s.update(bed=bed, G=_pinned((n, n)), freqs=_pinned(m, torch.float32),
                     xx=_pinned((n, n), torch.int32) if case["counts"] else None)
        elif kind == "ginv":
            _grm_call(h, bed, n, m)
            s.update(out=_pinned((n, n)))
        else:
            shape = (case["nvec"],) if case["nvec"] > 1 else ()
            s.update(dg=cb.DeviceGenotypes(bed, n, m, h), v=rng.normal(size=(n,) + shape),
                     w=rng.normal(size=(m,) + shape))
    elif kind in ("hinv", "final"):
        sire, dam = _pedigree(case, seed)
        _, _, G, gmap = _relationships(case, sire, dam, seed, torch.float64)
        y, aid, rows, p = _records(rng, _ped_values(rng, sire, dam, case["per"]), case.get("levels", 2))
        mme = cb.DeviceMME(h, y, aid, rows, p, sire.size)
        s.update(sire=sire, dam=dam, gmap=gmap, G=_host(G), mme=mme)
        if kind == "final":
            cb.ssgblup_qinv(mme, dam, sire, gmap, s["G"])
        else:
            s.update(A22=_pinned((gmap.size, gmap.size)), Gd=_pinned((gmap.size, gmap.size)))
    elif kind == "ssem":
        sire, dam = _pedigree(case, seed)
        csr, A22, G, gmap = _relationships(case, sire, dam, seed, torch.float32)
        Gd = _host((_inv32(0.95 * _tune(G, A22) + 0.05 * A22) - _inv32(A22)).double())
        del A22, G
        y, aid, rows, p = _records(rng, _ped_values(rng, sire, dam, case["per"]), case["levels"])
        s["mme"] = cb.DeviceMME(h, y, aid, rows, p, sire.size)
        s["mme"].set_qinv_split(*csr, Gd, gmap)
    elif kind in ("em", "solve", "dense"):
        G, (y, aid, rows, p) = _phenotypes(case, seed, torch.float32 if kind == "em" else torch.float64)
        Q = _bent_inverse32(G) if kind == "em" else _bent64(G)
        s.update(rec=(y, aid, rows, p), Q=_host(Q))
        if kind != "dense":
            s["mme"] = cb.DeviceMME(h, y, aid, rows, p, case["n"])
            s["mme"].set_qinv_dense(s.pop("Q"))
        if kind == "solve":
            B = rng.choice([-1.0, 1.0], size=(p + case["n"], case["nrhs"]))
            B[:p] = 0.0
            B[:, 0] = _wty(y, rows, p)
            s["B"] = B
    elif kind == "batch":
        s["problems"] = []
        for i in range(case["nprob"]):
            # sizes spread over [n_lo, n_hi] by their logarithm, the same for every seed
            n = int(round(case["n_lo"] * (case["n_hi"] / case["n_lo"]) ** (i / max(1, case["nprob"] - 1))))
            bed = _bed(_calls(_gen(100 * seed + i), n, case["m"]))
            y, aid, rows, p = _records(rng, rng.normal(size=n) * 0.6, 10)
            s["problems"].append(cb.BatchProblem(bed=bed, n=n, m=case["m"], y=y, aid=aid, rows=rows, p=p))
    elif kind == "mt":
        n, m = case["n"], case["m"]
        _grm_call(h, _bed(_calls(_gen(seed), n, m)), n, m)
        cb.invert_psd(h, None, n, download=False)
        s["Y"], s["X"] = _mt_data(case, seed, _vanraden(_calls(_gen(seed), n, m), n, torch.float64))
    torch.cuda.empty_cache()
    return s


def _bent64(G):
    w, U = torch.linalg.eigh(G)
    return (U / w.clamp(min=max(1e-12 * float(w[-1]), 1e-6))) @ U.T


def _wty(y, rows, p):
    fp, fc, fv = rows
    out = np.zeros(p + y.size)
    np.add.at(out, fc, np.repeat(y, np.diff(fp)) * fv)
    out[p:] = y
    return out


def run(s):
    c, h = s["case"], s["h"]
    kind = c["kind"]
    if kind == "grm":
        s2pq, valid = _grm_call(h, s["bed"], c["n"], c["m"], s["G"], s["xx"], s["freqs"])
        out = {"G": s["G"], "freqs": s["freqs"], "sum2pq": s2pq, "valid": valid}
        return dict(out, xx=s["xx"]) if c["counts"] else out
    if kind == "ginv":
        h.check(cb.lib().cbx_invert_psd(h.raw, None, c["n"], c["ridge"], ptr(s["out"])))
        return s["out"]
    if kind == "hinv":
        gm = s["gmap"]
        h.check(cb.lib().cbx_ssgblup_qinv(h.raw, s["dam"].size, ptr(s["dam"]), ptr(s["sire"]), gm.size, ptr(gm),
                                          ptr(s["G"]), 0.05, 1, 1.0, 1.0, 0.0, ptr(s["A22"]), ptr(s["Gd"])))
        return {"A22": s["A22"], "Gd": s["Gd"]}
    if kind == "final":
        r = cb.final_solve(s["mme"], 0.35, 0.65, solver=1, tol=1e-13, precision=MIXED if c["mixed"] else FP64)
        return {k: r[k] for k in ("sol", "beta_se", "Cinv_beta")}
    if kind == "solve":
        X, _, _ = s["mme"].pcg_solve(1.5, s["B"], tol=1e-13, precision=MIXED if c["mixed"] else FP64)
        return X
    if kind == "dense":
        # a whole analysis: records and G^-1 in, variance components and breeding values out
        y, aid, rows, p = s["rec"]
        mme = cb.DeviceMME(h, y, aid, rows, p, c["n"])
        mme.set_qinv_dense(s["Q"])
        r = cb.AIREML(mme, *START, cb.RemlConfig.default(mode=MODE_AUTO))
        vu, ve = r.solve()
        return {"var": [vu, ve], "logL": r.history[-1]["logL"], "sol": r.solution}
    if kind == "em":
        r = cb.AIREML(s["mme"], *START, cb.RemlConfig.default(mode=MODE_EM, precision=MIXED, max_iter=3, pcg_tol=1e-12))
        vu, ve = r.solve()
        return {"var": [vu, ve], "trace": [x["trace"] for x in r.history], "sol": r.solution}
    if kind == "ssem":
        r = cb.AIREML(s["mme"], *START, cb.RemlConfig.default(mode=MODE_EM, precision=MIXED, pcg_tol=1e-12))
        it = [r.run_iteration(grad_probes=c["probes"], solution=True) for _ in range(3)]
        return {"var": [x[k] for x in it for k in ("var_u", "var_e")], "grad": [x["grad"] for x in it],
                "trace": [x["trace"] for x in it], "sol": r.solution}
    if kind == "snp":
        return {"zt_v": s["dg"].multiply_Zt_v(s["v"]), "z_w": s["dg"].multiply_Z_v(s["w"])}
    if kind == "batch":
        cfg = cb.RemlConfig.default(mode=MODE_EM, precision=MIXED, max_iter=3, pcg_tol=1e-12)
        res = cb.batch_reml(s["problems"], cfg, workers=1)
        return [[r.var_u, r.var_e, r.solution] for r in res]
    v = cb.MvEigenVce(h, cb.MvOptions())
    v.prepare(s["Y"], s["X"])
    v.runNullModel()
    r = cb.solve_multi_trait(h, s["Y"], s["X"], v.getVg(), v.getVe())
    return {"Vg": v.getVg(), "Ve": v.getVe(), "beta": r["beta"], "u": r["u"]}


def work(case):
    """Inputs once, outputs once; the operations of the method itself, with 40 operator products a solve."""
    k, f = case["kind"], 8.0
    n, m = case.get("n", 0), case.get("m", 0)
    if k == "grm":
        return {"bytes": n * m / 4 + n * n * (f + 4 * case["counts"]), "flops": 1.0 * n * n * m}
    if k == "ginv":
        return {"bytes": 2 * f * n * n, "flops": 1.0 * n ** 3}
    if k in ("hinv", "final", "ssem"):
        ng, q = case["per"] * case["gen_g"], case["per"] * case["gens"]
        if k == "hinv":
            return {"bytes": 3 * f * ng * ng, "flops": 2.0 * ng ** 3}
        nrhs = 1 + case["levels"] if k == "final" else 1 + max(32, case["probes"])
        return {"bytes": 4.0 * ng * ng + f * q * nrhs, "flops": 2.0 * ng * ng * nrhs * 40 * (3 if k == "ssem" else 1)}
    if k == "solve":
        return {"bytes": 4.0 * n * n + 2 * f * n * case["nrhs"], "flops": 2.0 * n * n * case["nrhs"] * 40}
    if k == "dense":  # six AI steps: inverse and factor of the LHS, P V; then logL
        return {"bytes": f * n * n, "flops": 6.0 * 3.3 * n ** 3}
    if k == "em":
        return {"bytes": 4.0 * n * n + f * n * 33, "flops": 3 * 2.0 * n * n * 33 * 40}
    if k == "snp":
        return {"bytes": n * m / 4 + 2 * f * (n + m) * case["nvec"], "flops": 4.0 * n * m * case["nvec"]}
    if k == "batch":
        r = (case["n_hi"] / case["n_lo"]) ** (1 / max(1, case["nprob"] - 1))
        ns = [case["n_lo"] * r ** i for i in range(case["nprob"])]
        return {"bytes": sum(x * m / 4 for x in ns), "flops": sum(x * x * m + x ** 3 + 240 * x * x * 33 for x in ns)}
    t = case["traits"]
    return {"bytes": 2 * f * n * n, "flops": 9.0 * n ** 3 + (n * t) ** 3 / 3.0}


# ---- plain 64-bit values ------------------------------------------------------
def _solve64(Q, y, rows, p, lam, B):
    """LHS(lam)^-1 B with one record an animal in order, dense."""
    X = _dense_design(y, rows, p)
    n = y.size
    M = torch.zeros(p + n, p + n, dtype=torch.float64, device="cuda")
    M[:p, :p], M[:p, p:], M[p:, :p] = X.T @ X, X.T, X
    M[p:, p:] = lam * Q
    M.diagonal()[p:] += 1.0
    return torch.cholesky_solve(B, torch.linalg.cholesky(M))


def _dense_design(y, rows, p):
    fp, fc, fv = rows
    X = np.zeros((y.size, p))
    X[np.repeat(np.arange(y.size), np.diff(fp)), fc] = fv
    return torch.from_numpy(X).cuda()


def exact(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed + 21)
    if kind == "grm" and case["n"] ** 2 * case["m"] < 3e12:
        n, m = case["n"], case["m"]
        G = _vanraden(_calls(_gen(seed), n, m), n, torch.float64)
        st = [_centre(x, torch.float32)[1:] for _, x in _calls(_gen(seed), n, m)]
        f = torch.cat([torch.where(k, f, -1.0) for _, f, k in st])
        out = {"G": G, "freqs": f, "sum2pq": float(sum(float(w.sum()) for w, _, _ in st)), "valid": None}
        return dict(out, xx=None) if case["counts"] else out
    if kind == "ginv":
        n = case["n"]
        G = _vanraden(_calls(_gen(seed), n, case["m"]), n, torch.float64)
        G.diagonal().add_(case["ridge"])
        return _bent64(G)
    if kind in ("hinv", "final"):
        sire, dam = _pedigree(case, seed)
        csr, A22, G, gmap = _relationships(case, sire, dam, seed, torch.float64)
        Gb = 0.95 * _tune(G, A22) + 0.05 * A22
        Gd = torch.linalg.inv(Gb) - torch.linalg.inv(A22)
        if kind == "hinv":
            return {"A22": A22, "Gd": Gd}
        y, aid, rows, p = _records(rng, _ped_values(rng, sire, dam, case["per"]), case["levels"])
        q = sire.size
        ap, ac, av = (torch.from_numpy(x).cuda() for x in csr)
        Q = torch.zeros(q, q, dtype=torch.float64, device="cuda")
        Q[torch.repeat_interleave(torch.arange(q, device="cuda"), ap.diff()), ac.long()] = av
        Q[int(gmap[0]):, int(gmap[0]):] += Gd
        B = torch.zeros(p + q, 1 + p, dtype=torch.float64, device="cuda")
        B[:, 0] = torch.from_numpy(_wty(y, rows, p)).cuda()
        B[:p, 1:] = torch.eye(p, dtype=torch.float64, device="cuda")
        S = _solve64(Q, y, rows, p, 0.65 / 0.35, B)
        Ci = S[:p, 1:]
        return {"sol": S[:, 0], "beta_se": (0.65 * Ci.diagonal()).sqrt(), "Cinv_beta": Ci}
    if kind == "solve":
        G, (y, aid, rows, p) = _phenotypes(case, seed, torch.float64)
        B = rng.choice([-1.0, 1.0], size=(p + case["n"], case["nrhs"]))
        B[:p] = 0.0
        B[:, 0] = _wty(y, rows, p)
        return _solve64(_bent64(G), y, rows, p, 1.5, torch.from_numpy(B).cuda())
    if kind == "dense":
        return _dense_reml64(case, seed)
    if kind == "snp":
        n, m, k = case["n"], case["m"], case["nvec"]
        shape = (k,) if k > 1 else ()
        v = torch.from_numpy(rng.normal(size=(n,) + shape)).cuda().reshape(n, k)
        w = torch.from_numpy(rng.normal(size=(m,) + shape)).cuda().reshape(m, k)
        zt, zw = [], torch.zeros(n, k, dtype=torch.float64, device="cuda")
        for j, x in _calls(_gen(seed), n, m):
            for i in range(0, x.shape[0], 512):
                b = x[i:i + 512]
                ok = b >= 0
                mu = torch.where(ok, b, 0).sum(1, dtype=torch.float64) / ok.sum(1)
                var = mu * (1 - mu / 2)
                inv = torch.where(var < 1e-9, 0.0, var.rsqrt())
                z = torch.where(ok, (b.double() - mu[:, None]) * inv[:, None], 0.0)
                zt.append(z @ v)
                zw += z.T @ w[j + i:j + i + 512]
        return {"zt_v": torch.cat(zt).reshape((m,) + shape), "z_w": zw.reshape((n,) + shape)}
    return None


def _dense_reml64(case, seed):
    """Dense AI-REML: Newton steps with the exact average information, halved until logL rises."""
    G, (y, aid, rows, p) = _phenotypes(case, seed, torch.float64)
    Q = _bent64(G)
    n = case["n"]
    V = torch.cholesky_inverse(torch.linalg.cholesky(Q))
    logdet_v = -2.0 * torch.linalg.cholesky(Q).diagonal().log().sum()
    X, yt = _dense_design(y, rows, p), torch.from_numpy(y).cuda()
    W = torch.cat([X, torch.eye(n, dtype=torch.float64, device="cuda")], 1)

    def at(vu, ve):
        M = W.T @ W
        M[p:, p:] += ve / vu * Q
        L = torch.linalg.cholesky(M)
        sol = torch.cholesky_solve((W.T @ yt)[:, None], L)[:, 0]
        e = yt - W @ sol
        ll = -0.5 * (2 * L.diagonal().log().sum() + (n - p - n) * math.log(ve) + n * math.log(vu) + yt @ e / ve
                     + logdet_v)
        return L, sol, e, float(ll)

    vu, ve = START
    ll, sol = None, None
    for _ in range(20):
        L, sol, e, cur = at(vu, ve)
        P = (torch.eye(n, dtype=torch.float64, device="cuda") - W @ torch.cholesky_solve(W.T, L)) / ve
        M = P @ V
        t = float((M * P).sum())
        AI = 0.5 * np.array([[float((M * M.T).sum()), t], [t, float((P * P).sum())]])
        Py = e / ve
        g = 0.5 * np.array([float(Py @ (V @ Py) - M.trace()), float(Py @ Py - P.trace())])
        d = np.linalg.solve(AI, g)
        old = (vu, ve)
        for k in range(6):
            if vu + d[0] > 0 and ve + d[1] > 0:
                new = at(vu + d[0], ve + d[1])[3]
                if new > cur or k == 5:
                    vu, ve = vu + d[0], ve + d[1]
                    ll = new
                    break
            d = d / 2
        else:
            return None
        if abs(vu - old[0]) + abs(ve - old[1]) < 1e-4:
            break
    return {"var": [vu, ve], "logL": ll, "sol": sol}
