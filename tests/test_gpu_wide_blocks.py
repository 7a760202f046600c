"""Blocks in which every trait has its own missingness pattern, with SNP
columns that nearly equal a covariate: D - A'A keeps 1 / kappa of D, and the
covariate projections A must be summed as accurately as the row gathers did.
Both forms and the zero-allocation scan against the FP64 oracle.
"""
import functools

import numpy as np
import pytest

from omicabelnomm_b200 import engine as E
from omicabelnomm_b200 import synth
from test_gpu_parity import T_ABS, T_REL, engine_run, oracle_dense
from test_zz_no_alloc import noalloc_dense

pytestmark = pytest.mark.gpu

SPREAD = 0.02                       # of the columns about the covariate, whose own is 1
KAPPA = 1.0 + 1.0 / SPREAD ** 2     # 2,501


@functools.lru_cache(maxsize=None)
def _data(n, l, r, t=70):
    ds = synth.generate(synth.scaled(0, n=n, m=40, t=t, l=l, r=r, seed=700 + n + l))
    rng = np.random.Generator(np.random.PCG64(n + l + r))
    for c in range(0, ds.XR.shape[0], r):           # the SNP's first column, its second stays a dosage
        ds.XR[c] = ds.XL[l - 1] + SPREAD * rng.standard_normal(n)
    if r == 2:
        ds.XR[1::2] = np.clip(rng.binomial(2, 0.3, (40, n)) + rng.uniform(-0.05, 0.05, (40, n)), 0, 2)
    res, _, _ = oracle_dense(ds, r)
    assert not res.dense.singular.any()
    return ds, res


def _check(ds, res, dense):
    t_ref = np.abs(res.dense.tstat[:, :, res.l:])
    # FP32 sums keep 2^-24 of D and A: two of each, on both sides of a difference 1 / kappa of them
    lim = (T_REL + 2.0 ** -22 * KAPPA) * t_ref.max(2, keepdims=True) + T_ABS
    dt = np.abs(dense[2] - t_ref)
    assert np.all(dt <= lim), f"max |dt| {dt.max():.3g}, worst ratio {(dt / lim).max():.3g}"
    se_ref = res.dense.se[:, :, res.l:]
    assert np.all(np.abs(dense[1] - se_ref) <= (1e-4 + 2.0 ** -22 * KAPPA) * se_ref)


CASES = [(1500, 4, 1), (1501, 4, 2), (5003, 4, 1), (9973, 4, 1), (9973, 4, 2), (1500, 9, 1), (16384, 4, 1),
         (16386, 9, 1)]


@pytest.mark.parametrize("n,l,r", CASES)
def test_columns_near_a_covariate(n, l, r):
    ds, res = _data(n, l, r)
    eng, _, dense = engine_run(ds, r)
    assert eng.tuning()["stats_path"] == 1
    eng.close()
    _check(ds, res, dense)


@pytest.mark.parametrize("n,l,r", CASES)
def test_columns_near_a_covariate_mixed(n, l, r, monkeypatch):
    """The mixed form's own product X'y~ (BF16) is the largest error here; the covariate sums must add nothing
    to what it leaves with the row gathers."""
    ds, res = _data(n, l, r)
    t_ref, se_ref = np.abs(res.dense.tstat[:, :, res.l:]), res.dense.se[:, :, res.l:]
    err = {}
    for path in ("", "gather"):
        if path:
            monkeypatch.setenv("OA_STATS_PATH", path)
        eng, _, dense = engine_run(ds, r, precision=E.MIXED)
        assert eng.tuning()["stats_path"] == (2 if path else 1)
        eng.close()
        err[path] = np.linalg.norm(dense[2] - t_ref), np.linalg.norm(dense[1] - se_ref)
        assert np.all(np.abs(dense[1] - se_ref) <= (1e-4 + 2.0 ** -22 * KAPPA) * se_ref)
    assert err[""][0] <= 1.25 * err["gather"][0]


@pytest.mark.parametrize("n,l,r", [(1500, 4, 1), (1501, 4, 2), (1500, 9, 1), (5003, 4, 1)])
def test_columns_near_a_covariate_noalloc(n, l, r):
    ds, res = _data(n, l, r)
    _check(ds, res, noalloc_dense(ds, r))


@pytest.mark.parametrize("prec", [E.PLAIN, E.MIXED])
@pytest.mark.parametrize("l,r", [(4, 1), (10, 2)])
def test_wide_block_paths(l, r, prec):
    """One column per SNP takes the pre-GEMM, two with more than eight covariates the row gathers; both within
    the bars, and the same whatever was asked for before."""
    ds = synth.generate(synth.scaled(0, n=700, m=60, t=60, l=l, r=r, seed=760 + l))
    res, _, _ = oracle_dense(ds, r)
    t_ref = np.abs(res.dense.tstat[:, :, res.l:])
    got = {}
    for path in (0, 1, 2):
        eng = E.Engine(700, l, r, 60, 60, precision=prec, store_all=True, min_t_store=1.6, min_r2_store=1e-6)
        eng.set_covariates(ds.XL)
        eng.set_traits(ds.Y)
        eng.set_tuning(stats_path=path)          # after the traits
        eng.enable_dense(True)
        eng.run(ds.XR)
        got[path] = eng.dense(60)
        if path == 0:
            assert eng.tuning()["stats_path"] == (1 if r == 1 else 2)
        eng.close()
        lim = T_REL * t_ref.max(2, keepdims=True) + T_ABS if prec == E.PLAIN else 1e-3
        assert np.all(np.abs(got[path][2] - t_ref) <= lim)
    for a, b in zip(got[0], got[1 if r == 1 else 2]):
        np.testing.assert_array_equal(a, b)
