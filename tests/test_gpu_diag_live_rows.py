"""diag K over the markers that count: the sums of a handle with markers left out are those of
a handle without them, to the bit, and so are the fits that precondition with it.

The markers are summed in ranges of at least 64; the sizes put the left-out ones inside and at
the edges of the ranges, and of the blocks of 1,024 rows in which they are listed."""
import numpy as np
import pytest

import csaige_b200 as cs
import oracle_ffi as O

pytestmark = pytest.mark.gpu


def _config(**kw):
    return cs.AiRemlConfig(max_iter=4, precision=cs.PREC_MIXED, solve=cs.SOLVE_BLOCK,
                           warm_start=cs.WARM_RECYCLED, precond=cs.PRECOND_DIAG_K, **kw)


def _cohort(n, m, **kw):
    spec = cs.CohortSpec(n=n, m=m, seed=29, prevalence=0.25, h2=0.4, n_covar=2, **kw)
    bed = cs.gen_bed(spec)
    af, mac, nv = O.marker_stats(bed, n, m)
    return spec, bed, af, np.nonzero((af >= 0.01) & (af <= 0.99))[0]


def _grm(c, idx, af=None):
    spec, bed, afs, _ = c
    return cs.OnTheFlyGrm.from_bed(bed, spec.n, spec.m, idx, (afs if af is None else af)[idx],
                                   precision=cs.PREC_MIXED)


@pytest.mark.parametrize("n,m", [(700, 900), (4200, 3300)])
def test_mixed_loco_with_the_exact_diagonal_equals_the_refit(n, m):
    c = _cohort(n, m)
    y, x = cs.gen_pheno(c[0])
    keep = c[3]
    # a chromosome of every third marker, one of a few, one run of neighbours
    k = np.arange(len(keep))
    names = np.where(k % 3 == 0, "1", np.where(k < 40, "2", np.where(k < 450, "3", "4")))
    res = cs.run_loco(y, x, _grm(c, keep), list(names), cs.TraitType.Binary, _config())
    for chrom, r in res.items():
        ref = cs.fit_ai_reml(y, x, _grm(c, keep[names != chrom]), cs.TraitType.Binary, _config())
        assert np.array_equal(r.tau, ref.tau), chrom
        assert np.array_equal(r.mu, ref.mu), chrom
        assert np.array_equal(r.alpha, ref.alpha), chrom


@pytest.mark.parametrize("m,dead", [(300, [0]), (1024, [1023]), (1025, [1024]), (2500, range(0, 2500, 7)),
                                    (2500, range(64, 1100)), (130, range(130))])
def test_diagonal_without_constant_markers(m, dead):
    # a marker of frequency 0 has no standardised column
    n = 3001
    c = _cohort(n, m, missing_rate=0.02)
    every, dead = np.arange(m), np.array(list(dead))
    af = np.clip(c[2], 0.02, 0.98)
    gone = af.copy()
    gone[dead] = 0.0
    rest = np.setdiff1d(every, dead)
    got = _grm(c, every, gone).diag() * m  # over all rows of the handle, the constant ones too
    if not len(rest):
        assert np.array_equal(got, np.zeros(n))
        return
    z = O.standardize(O.dosages(c[1], n, rest), af[rest], 0)
    want = (z * z).sum(axis=0)
    # sums of at most m non-negative terms, each within a few units of rounding
    np.testing.assert_allclose(got, want, rtol=1e-15 * (m + 10), atol=0)


@pytest.mark.parametrize("subset", [False, True])
def test_pinned_upload_with_the_exact_diagonal_gives_the_same_fit(subset):
    # the streamed build keeps the variance-ratio candidates as rows of the handle that do not
    # count
    import torch
    n, m = 1500, 2500
    spec = cs.CohortSpec(n=n, m=m, seed=31, missing_rate=0.02, prevalence=0.2, h2=0.3, n_covar=2)
    bed = cs.gen_bed(spec)
    y, x = cs.gen_pheno(spec)
    sidx = None
    if subset:
        sidx = np.sort(np.random.default_rng(3).choice(n, 1201, replace=False))
        y, x = y[sidx], x[sidx]
    pinned = torch.empty(bed.size, dtype=torch.uint8, pin_memory=True)
    pinned.numpy()[:] = bed
    kw = dict(sample_idx=sidx, min_maf=0.05, variance_ratio=True)
    a = cs.fit_null_from_bed(bed, n, m, y, x, cs.TraitType.Binary, _config(), **kw)
    b = cs.fit_null_from_bed(pinned.numpy(), n, m, y, x, cs.TraitType.Binary, _config(), **kw)
    assert np.array_equal(a.ai_reml.tau, b.ai_reml.tau)
    assert np.array_equal(a.ai_reml.alpha, b.ai_reml.alpha)
    assert np.array_equal(a.ai_reml.mu, b.ai_reml.mu)
