"""The work that a user of this library has it do, as cases that can be timed and checked.

Each case goes through the public Python API (csaige_b200), over the real range of
cohort sizes: from the CPU-scale cohort (2,000 samples, 5,000 markers), where launches
and latency count, to a biobank cohort (200,000 samples, 150,000 markers), with sample
and marker counts that are no multiples of any tile.

  product     K v for one vector or a block of vectors (both precisions, host and
              device buffers)
  pcg         solves with Sigma = tau0 W^-1 + tau1 K for a block of right-hand sides
  fit         an AI-REML null-model fit on a GRM handle
  loco        the leave-one-chromosome-out refits on a GRM handle
  genotypes   from a .bed in device memory to a GRM handle: marker statistics, QC and
              marker split, the handle, its diagonal
  fit_null    the whole fit-null call from a .bed in (pinned) host memory, with the
              variance ratio
  sparse_grm  the explicit relatedness matrix of create-sparse-grm

Inputs are the seeded synthetic cohorts of the library's own generator: allele
frequencies U(0.01, 0.5), Hardy-Weinberg genotypes, sibling and cousin pairs, calls
missing at random.
"""
import math

import numpy as np
import torch

import csaige_b200 as cs
from csaige_b200 import api

FIT_TOL = 1e-5  # the fit-null command's tolerance of tau


def listed():
    return [
        # one K v of the CPU-scale cohort from host arrays at the default precision: the
        # smallest call a score-test or a PCG of the caller's own makes
        dict(name="product_small", kind="product", n=2000, m=5000, nrhs=1, precision="fp32",
             host=True, missing=0.01),
        # a few vectors in the plain (FP32) arithmetic, ragged sizes, on the device
        dict(name="product_fp32_block", kind="product", n=20011, m=30001, nrhs=6,
             precision="fp32", host=False, missing=0.01),
        # one vector, tensor-core precision, biobank cohort: each PCG step of an AI solve
        dict(name="product_one_large", kind="product", n=200000, m=150000, nrhs=1,
             precision="mixed", host=False, missing=0.01),
        # the block of a fit (y, covariates and probes) at the mid-size cohort
        dict(name="product_block", kind="product", n=50000, m=100000, nrhs=37,
             precision="mixed", host=False, missing=0.01),
        # a block solve from host arrays, as a caller with its own weights makes it
        dict(name="pcg_block", kind="pcg", n=12007, m=25013, nrhs=31, precision="mixed",
             missing=0.02),
        # the CPU-scale binary-trait fit with the default configuration (FP32 products,
        # one PCG per right-hand side, zero starts)
        dict(name="fit_small_default", kind="fit", n=2000, m=5000, trait="binary",
             covariates=2, config="default", missing=0.01),
        # the same cohort with the fast configuration
        dict(name="fit_small_fast", kind="fit", n=2000, m=5000, trait="binary",
             covariates=2, config="fast", missing=0.01),
        # a biobank fit, fast configuration: binary trait of 2 % prevalence
        dict(name="fit_large", kind="fit", n=200000, m=150000, trait="binary", covariates=10,
             config="fast", missing=0.01),
        # 22 chromosome refits of a quantitative trait
        dict(name="loco_22", kind="loco", n=9001, m=22003, chroms=22, covariates=4,
             missing=0.01),
        # handle set-up for a sub-cohort of a biobank .bed that already is in device memory
        dict(name="genotypes_subset", kind="genotypes", n_fam=150001, n=60013, m=40000,
             missing=0.02),
        # the whole command's genotype part from host memory, variance ratio included
        dict(name="fit_null_host", kind="fit_null", n=20000, m=50000, trait="binary",
             covariates=6, missing=0.01),
        # create-sparse-grm on a cohort of a few thousand samples
        dict(name="sparse_grm", kind="sparse_grm", n=4001, m=6007, missing=0.01),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["product", "product", "product", "pcg", "fit", "fit", "loco",
                       "genotypes", "fit_null", "sparse_grm"])
    missing = rng.choice([0.0, 0.005, 0.01, 0.01, 0.02, 0.05])
    if kind == "product":
        mixed = rng.random() < 0.7
        n = _log_int(rng, 1000, 200000)
        m = _log_int(rng, 500, 150000)
        nrhs = rng.choice([1, 1, 2, 5, 13, 31, 41, 42, 50]) if mixed else rng.choice([1, 1, 3, 8])
        return dict(kind=kind, n=n, m=m, nrhs=nrhs, precision="mixed" if mixed else "fp32",
                    host=rng.random() < 0.3 and n * nrhs < 300000, missing=missing)
    if kind == "pcg":
        return dict(kind=kind, n=_log_int(rng, 1000, 16000), m=_log_int(rng, 2000, 40000),
                    nrhs=rng.choice([1, 3, 11, 31, 41]), precision=rng.choice(["mixed", "mixed", "fp32"]),
                    missing=missing)
    if kind == "fit":
        if rng.random() < 0.3:
            return dict(kind=kind, n=_log_int(rng, 1500, 4000), m=_log_int(rng, 3000, 8000),
                        trait=rng.choice(["binary", "quantitative"]), covariates=rng.randint(1, 4),
                        config="default", missing=missing)
        n = _log_int(rng, 2000, 100000)
        return dict(kind=kind, n=n, m=_log_int(rng, 5000, 100000),
                    trait=rng.choice(["binary", "binary", "quantitative"]),
                    covariates=rng.randint(1, 10), config="fast", missing=missing)
    if kind == "loco":
        return dict(kind=kind, n=_log_int(rng, 2000, 12000), m=_log_int(rng, 5000, 25000),
                    chroms=rng.choice([5, 10, 22]), covariates=rng.randint(1, 6), missing=missing)
    if kind == "genotypes":
        n_fam = _log_int(rng, 2000, 200000)
        n = n_fam if rng.random() < 0.4 else max(1000, int(n_fam * rng.uniform(0.3, 0.95)))
        return dict(kind=kind, n_fam=n_fam, n=n, m=_log_int(rng, 2000, 60000), missing=missing)
    if kind == "fit_null":
        return dict(kind=kind, n=_log_int(rng, 2500, 30000), m=_log_int(rng, 6000, 60000),
                    trait=rng.choice(["binary", "quantitative"]), covariates=rng.randint(1, 8),
                    missing=missing)
    return dict(kind=kind, n=_log_int(rng, 500, 4500), m=_log_int(rng, 2000, 6000), missing=missing)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _spec(case, seed, n=None):
    quantitative = case.get("trait") == "quantitative" or case["kind"] == "loco"
    n = n or case["n"]
    return cs.CohortSpec(
        seed=1000003 + seed, n=n, m=case["m"], sib_frac=0.10, cousin_frac=0.02,
        missing_rate=case["missing"], maf_lo=0.01, maf_hi=0.5,
        trait=int(cs.TraitType.Quantitative if quantitative else cs.TraitType.Binary),
        n_covar=case.get("covariates", 2), prevalence=0.10 if n < 50000 else 0.02,
        h2=0.3 if quantitative else 0.2)


def _bed_dev(spec):
    bed = torch.empty(spec.bed_len, dtype=torch.uint8, device="cuda")
    cs.gen_bed_dev(spec, bed.data_ptr())
    return bed


def _handle(spec, precision):
    """A GRM handle over the cohort's QC-passing GRM markers, as fit-null builds it."""
    bed = _bed_dev(spec)
    af, mac, nv = api.bed_marker_stats_dev(bed.data_ptr(), spec.bed_len, spec.n, spec.m)
    idx, _ = cs.select_grm_markers(af, mac, nv, spec.n)
    grm = cs.OnTheFlyGrm.from_bed_dev(bed.data_ptr(), spec.bed_len, spec.n, spec.m, idx, af[idx],
                                      precision=precision)
    return grm, idx


def _precision(name):
    return cs.PREC_MIXED if name == "mixed" else cs.PREC_FP32


def _vectors(case, seed):
    """What a PCG multiplies: normal vectors with, in a block, a few +-1 probes."""
    g = torch.Generator(device="cuda").manual_seed(77 + seed)
    v = torch.randn(case["nrhs"], case["n"], generator=g, device="cuda", dtype=torch.float64)
    if case["nrhs"] > 2:
        v[1::2] = torch.sign(v[1::2])
    return v


def _weights(case, seed):
    """Working weights mu (1 - mu) of a binary trait."""
    g = torch.Generator(device="cuda").manual_seed(78 + seed)
    mu = torch.sigmoid(0.5 * torch.randn(case["n"], generator=g, device="cuda",
                                         dtype=torch.float64) - 2.0)
    return mu * (1 - mu)


def _subset(case, seed):
    if case["n"] == case["n_fam"]:
        return None
    r = np.random.default_rng(79 + seed)
    return np.sort(r.choice(case["n_fam"], case["n"], replace=False)).astype(np.int64)


def _config(name):
    if name == "default":
        return cs.AiRemlConfig()
    return cs.AiRemlConfig(tol=FIT_TOL, precision=cs.PREC_MIXED, solve=cs.SOLVE_BLOCK,
                           warm_start=cs.WARM_RECYCLED)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "product":
        v = _vectors(case, seed)
        grm, _ = _handle(_spec(case, seed), _precision(case["precision"]))
        if case["host"]:
            a = v.cpu().numpy()
            return dict(case=case, grm=grm, v=a[0].copy() if case["nrhs"] == 1 else a)
        return dict(case=case, grm=grm, v=v, out=torch.empty_like(v))
    if kind == "pcg":
        grm, _ = _handle(_spec(case, seed), _precision(case["precision"]))
        return dict(case=case, grm=grm, solver=cs.PcgSolver(), w=_weights(case, seed).cpu().numpy(),
                    tau=np.array([1.0, 0.35]), b=_vectors(case, seed).cpu().numpy())
    if kind in ("fit", "loco"):
        spec = _spec(case, seed)
        y, x = cs.gen_pheno(spec)
        s = dict(case=case, y=y, x=x, trait=cs.TraitType(spec.trait))
        if kind == "fit":
            s["config"] = _config(case["config"])
            s["grm"], _ = _handle(spec, s["config"].precision)
        else:
            s["config"] = _config("fast")
            s["grm"], idx = _handle(spec, s["config"].precision)
            c = idx * case["chroms"] // case["m"] + 1  # neighbouring markers share one
            s["chroms"] = ["chr%02d" % k for k in c]
        return s
    if kind == "genotypes":
        spec = _spec(case, seed, n=case["n_fam"])
        return dict(case=case, bed=_bed_dev(spec), bed_len=spec.bed_len, sidx=_subset(case, seed))
    spec = _spec(case, seed)
    bed = torch.empty(spec.bed_len, dtype=torch.uint8, pin_memory=True)
    bed.copy_(_bed_dev(spec))
    s = dict(case=case, pinned=bed, bed=bed.numpy())
    if kind == "fit_null":
        s["y"], s["x"] = cs.gen_pheno(spec)
        s["trait"] = cs.TraitType(spec.trait)
        s["config"] = _config("fast")
        s["vr"] = cs.VarianceRatioConfig(precision=cs.PREC_MIXED)
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "product":
        if case["host"]:
            return s["grm"].mat_vec(s["v"])
        s["grm"].mat_vec_dev(s["v"].data_ptr(), s["out"].data_ptr(), case["nrhs"])
        return s["out"]
    if kind == "pcg":
        r = s["solver"].solve(s["grm"], s["w"], s["tau"], s["b"])
        r = r if isinstance(r, list) else [r]
        return dict(x=np.stack([c.x for c in r]), iterations=np.array([c.iterations for c in r]))
    if kind == "fit":
        f = cs.fit_ai_reml(s["y"], s["x"], s["grm"], s["trait"], s["config"])
        return dict(tau=f.tau, tau_trace=_padded(f.tau_trace.ravel(), 60), alpha=f.alpha, mu=f.mu,
                    eta=f.eta, weights=f.working_weights, log_likelihood=f.log_likelihood,
                    iterations=f.iterations)
    if kind == "loco":
        f = cs.run_loco(s["y"], s["x"], s["grm"], s["chroms"], s["trait"], s["config"])
        k = sorted(f)
        return dict(tau=np.stack([f[c].tau for c in k]), alpha=np.stack([f[c].alpha for c in k]),
                    mu=np.stack([f[c].mu for c in k]))
    if kind == "genotypes":
        n, n_fam, m, ptr = case["n"], case["n_fam"], case["m"], s["bed"].data_ptr()
        af, mac, nv = api.bed_marker_stats_dev(ptr, s["bed_len"], n_fam, m, s["sidx"])
        idx, vr = cs.select_grm_markers(af, mac, nv, n)
        grm = cs.OnTheFlyGrm.from_bed_dev(ptr, s["bed_len"], n_fam, m, idx, af[idx],
                                          sample_idx=s["sidx"], precision=cs.PREC_MIXED)
        d = grm.diag()
        grm.close()
        return dict(af=af, mac=mac, n_valid=nv, split=_split(m, idx, vr), diagonal=d)
    if kind == "fit_null":
        f = cs.fit_null_from_bed(s["bed"], case["n"], case["m"], s["y"], s["x"], s["trait"],
                                 s["config"], variance_ratio=True, vr_config=s["vr"])
        a = f.ai_reml
        return dict(tau=a.tau, tau_trace=_padded(a.tau_trace.ravel(), 60), alpha=a.alpha, mu=a.mu,
                    iterations=a.iterations, m_grm=f.m_grm, m_vr=f.m_vr,
                    variance_ratio=f.variance_ratio.variance_ratio,
                    vr_markers=f.variance_ratio.n_markers_used)
    g, used = cs.compute_sparse_grm(s["bed"], case["n"], case["m"])
    k = 4 * case["n"]
    return dict(rows=_padded(g.rows, k), cols=_padded(g.cols, k), vals=_padded(g.vals, k),
                markers=used)


def _padded(a, k):
    """a in an array of k entries (how many there are depends on the data)."""
    out = np.zeros(max(k, a.size), a.dtype)
    out[:a.size] = a
    return out


def _split(m, idx, vr):
    """1 for a GRM marker, 2 for a variance-ratio candidate, 0 for a marker left out."""
    s = np.zeros(m, np.int8)
    s[idx] = 1
    s[vr] = 2
    return s


def work(case):
    """The packed genotypes once, the vectors in and out once; the multiply-adds of the
    products that no method saves (for a fit or a solve: one product of every column)."""
    n, m, kind = case["n"], case["m"], case["kind"]
    packed = m * ((n + 3) // 4)
    if kind in ("product", "pcg"):
        return dict(bytes=packed + 16 * n * case["nrhs"], flops=4 * n * m * case["nrhs"])
    if kind == "fit" or kind == "fit_null":
        q = 31 + 1 + case["covariates"]
        return dict(bytes=packed + 8 * n * (q + 4), flops=4 * n * m * q)
    if kind == "loco":
        q = 31 + 1 + case["covariates"]
        return dict(bytes=case["chroms"] * (packed + 8 * n * (q + 4)),
                    flops=4 * n * m * q * case["chroms"])
    if kind == "genotypes":
        return dict(bytes=m * ((case["n_fam"] + 3) // 4) + packed + 8 * n + 24 * m, flops=2 * n * m)
    return dict(bytes=packed + 4 * n * n, flops=n * (n + 1) * m)


# ---------------------------------------------------------------------------
# the same values in 64 bits, by plain torch
# ---------------------------------------------------------------------------
def _dosages(bed, n_fam, j0, j1, sidx=None):
    """Dosages (copies of the first allele, NaN for a missing call) of markers j0 .. j1-1."""
    bpm = (n_fam + 3) // 4
    rows = bed[3 + j0 * bpm:3 + j1 * bpm].view(j1 - j0, bpm)
    codes = torch.stack([(rows >> k) & 3 for k in (0, 2, 4, 6)], dim=2).view(j1 - j0, 4 * bpm)
    codes = codes[:, :n_fam] if sidx is None else codes[:, sidx]
    lut = torch.tensor([2.0, float("nan"), 1.0, 0.0], dtype=torch.float64, device=bed.device)
    return lut[codes.long()]


def _chunk(n):
    return max(16, int(1.0e8 / n))


def _stats(bed, n_fam, m, sidx=None):
    alt = torch.empty(m, dtype=torch.float64, device="cuda")
    valid = torch.empty_like(alt)
    c = _chunk(n_fam)
    for j in range(0, m, c):
        g = _dosages(bed, n_fam, j, min(m, j + c), sidx)
        alt[j:j + c] = torch.nansum(g, dim=1)
        valid[j:j + c] = (~torch.isnan(g)).sum(dim=1)
    return alt, valid


def _standardised(bed, n_fam, af, markers, sidx=None):
    """Z by chunks of the given markers: (g - 2p) / sqrt(2p (1 - p)), a missing call 0."""
    keep = torch.zeros(af.numel(), dtype=torch.bool, device="cuda")
    keep[torch.as_tensor(markers, device="cuda")] = True
    c = _chunk(n_fam)
    for j in range(0, af.numel(), c):
        k = keep[j:j + c].nonzero().flatten()
        if not k.numel():
            continue
        p = af[j:j + c][k][:, None]
        z = _dosages(bed, n_fam, j, min(af.numel(), j + c), sidx)[k] - 2 * p
        yield torch.nan_to_num(z / torch.sqrt(2 * p * (1 - p)), nan=0.0)


def _grm_markers(alt, valid, n):
    """The marker split draws from a ChaCha8 stream: the list is taken as given."""
    af = torch.where(valid > 0, alt / (2 * valid), torch.zeros_like(alt))
    mac = torch.minimum(alt, 2 * valid - alt)
    idx, _ = cs.select_grm_markers(af.cpu().numpy(), mac.cpu().numpy(),
                                   valid.cpu().numpy().astype(np.int64), n)
    return af, mac, idx


def exact(case, seed):
    kind, n, m = case["kind"], case["n"], case["m"]
    if kind in ("fit", "loco", "fit_null"):
        return None  # seeded probes and stopping rules decide these values, not arithmetic alone
    if kind == "pcg" and n > 16000:
        return None
    if kind == "genotypes":
        sidx = _subset(case, seed)
        sidx = None if sidx is None else torch.from_numpy(sidx).cuda()
        bed = _bed_dev(_spec(case, seed, n=case["n_fam"]))
        alt, valid = _stats(bed, case["n_fam"], m, sidx)
        af, mac, idx = _grm_markers(alt, valid, n)
        d = torch.zeros(n, dtype=torch.float64, device="cuda")
        for z in _standardised(bed, case["n_fam"], af, idx, sidx):
            d += (z * z).sum(dim=0)
        return dict(af=af, mac=mac, n_valid=valid.long(), split=None,
                    diagonal=d / len(idx))
    spec = _spec(case, seed)
    bed = _bed_dev(spec)
    alt, valid = _stats(bed, n, m)
    if kind == "sparse_grm":
        af = alt / (2 * valid)
        idx = ((af >= 0.01) & (af <= 0.99) & (2 * af * (1 - af) >= 1e-10)).nonzero().flatten()
        k = torch.zeros(n, n, dtype=torch.float64, device="cuda")
        for z in _standardised(bed, n, af, idx):
            k.addmm_(z.T, z)
        k /= idx.numel()
        at = torch.triu((k.abs() >= 0.125) | torch.eye(n, dtype=torch.bool, device="cuda")).nonzero()
        vals = k[at[:, 0], at[:, 1]].cpu().numpy()
        return dict(rows=None, cols=None, vals=_padded(vals, 4 * n), markers=None)
    af, _, idx = _grm_markers(alt, valid, n)
    v = _vectors(case, seed)
    if kind == "product":
        out = torch.zeros_like(v)
        for z in _standardised(bed, n, af, idx):
            out.addmm_(v @ z.T, z)
        out /= len(idx)
        return out[0] if case["host"] and case["nrhs"] == 1 else out
    k = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    for z in _standardised(bed, n, af, idx):
        k.addmm_(z.T, z)
    k *= 0.35 / len(idx)
    k.diagonal().add_(1.0 / _weights(case, seed).clamp_min(1e-30))
    low = torch.linalg.cholesky(k)
    return dict(x=torch.cholesky_solve(v.T.contiguous(), low).T.contiguous(), iterations=None)
