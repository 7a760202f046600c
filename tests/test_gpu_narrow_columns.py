"""SNP columns whose spread is small against their mean (a rare variant coded
by the major allele, an expression level, a year of birth), in the plain form
and the zero-allocation scan, against the FP64 oracle.

The rows between n and the next multiple of 64 must not reach the products:
the FP16 scale of a column follows its centred norm, which says nothing about
the mean.  n = 1,024 has no such rows.
"""
import numpy as np
import pytest

import quirk_cases as QC
from omicabelnomm_b200 import synth
from test_gpu_parity import T_ABS, T_REL, engine_run, oracle_dense
from test_zz_no_alloc import noalloc_dense

pytestmark = pytest.mark.gpu

SIZES = [500, 1000, 1024, 4713, 9973]


def narrow_dataset(n, r):
    """24 SNPs of r columns of one kind, the kinds in turn; the odd rows of a column are observed in every
    trait, so that no system is singular."""
    m, t = 24, 6
    ds = (QC.multicol(r, 500 + n, n=n, m=m, t=t, n_patterns=2) if r > 2 else
          synth.generate(synth.scaled(0, n=n, m=m, t=t, l=4, r=r, miss_mode="patterns", n_patterns=2, seed=500 + n)))
    rng = np.random.Generator(np.random.PCG64(n + r))
    seen = np.nonzero(~np.isnan(ds.Y).any(0))[0]
    for c in range(m * r):
        kind = c // r % 5
        x = ds.XR[c]
        if kind == 0:       # dosage 2 everywhere but in one row
            x[:] = 2.0
            x[rng.choice(seen)] = 1.6
        elif kind == 1:     # in twenty rows
            x[:] = 2.0
            x[rng.choice(seen, 20, replace=False)] = 1.95
        elif kind == 2:
            x[:] = 12.0 + 0.05 * rng.standard_normal(n)
        elif kind == 3:     # (four such columns at a deviation of 10 are singular by the oracle's eigenvalue rule)
            x[:] = np.round(1955.0 + (10.0 if r < 4 else 25.0) * rng.standard_normal(n))
        else:               # mean / sd = 1,000
            x[:] = 30.0 + 0.03 * rng.standard_normal(n)
    return ds


def check_narrow(ds, r, dense, kappa=None):
    res, _, _ = oracle_dense(ds, r)
    D = res.dense
    assert not D.singular.any()
    b, se, tt, r2 = dense
    assert np.all(np.isfinite(tt)), f"{np.isnan(tt[..., 0]).sum()} tests lost"
    t_ref, se_ref = D.tstat[:, :, res.l:], D.se[:, :, res.l:]
    # the systems are differences of FP32 column sums: each term is rounded to 2^-24 of x^2, the difference
    # is the spread, so the sums keep 2^-24 (1 + mean^2 / var) of it; four such (two sums, two sides)
    x = ds.XR.astype(np.float64)
    if kappa is None:
        kappa = (1.0 + x.mean(1) ** 2 / x.var(1)).reshape(-1, r).max(1)[None, :, None]
    t_sys = np.abs(t_ref).max(2, keepdims=True)
    lim = (T_REL + 2.0 ** -22 * kappa) * t_sys + T_ABS
    dt = np.abs(tt - np.abs(t_ref))
    assert np.all(dt <= lim), f"max |dt| {dt.max():.3g}, worst ratio {(dt / lim).max():.3g}"
    assert np.all(np.abs(se - se_ref) <= (1e-4 + 2.0 ** -22 * kappa) * se_ref)


@pytest.mark.parametrize("r", [1, 2, 4])
@pytest.mark.parametrize("n", SIZES)
def test_narrow_columns_plain(n, r):
    ds = narrow_dataset(n, r)
    _, rows, dense = engine_run(ds, r)
    check_narrow(ds, r, dense)
    assert rows.singular == 0


@pytest.mark.parametrize("r", [1, 2, 4])
@pytest.mark.parametrize("n", SIZES)
def test_centred_sums_do_not_cancel(n, r):
    """With an intercept the sums are those of the centred columns: the bar of ordinary columns, whatever the
    mean."""
    ds = narrow_dataset(n, r)
    _, _, dense = engine_run(ds, r)
    check_narrow(ds, r, dense, kappa=0.0)
    check_narrow(ds, r, noalloc_dense(ds, r), kappa=0.0)


@pytest.mark.parametrize("r", [1, 2, 4])
@pytest.mark.parametrize("n", SIZES)
def test_narrow_columns_noalloc(n, r):
    ds = narrow_dataset(n, r)
    check_narrow(ds, r, noalloc_dense(ds, r))
