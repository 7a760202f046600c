"""SNP columns without centring (no intercept among the covariates) at
n = 10,000: own patterns (every trait its own) take the row gathers, whose
sums do not cancel as the pre-GEMM's; few patterns take the pre-GEMM (in the
mixed form with its BF16 sums, whose errors without centring reach 2e-3 of t
and are not asserted here).  Bars: the plain and mixed forms' of
tests/test_gpu_precision.py.
"""
import functools

import numpy as np
import pytest

from omicabelnomm_b200 import engine as E
from omicabelnomm_b200 import synth
from test_gpu_parity import T_ABS, T_REL, oracle_dense

pytestmark = pytest.mark.gpu


@functools.lru_cache(maxsize=None)
def _data(patterns, r):
    t = 70
    ds = synth.generate(synth.scaled(0, n=10000, m=40, t=t, l=5, r=r, seed=600 + r,
                                     **(dict(miss_mode="patterns", n_patterns=4) if patterns == "few" else {})))
    ds.XL = np.ascontiguousarray(ds.XL[1:])          # sex, age and the components: no intercept
    res, _, _ = oracle_dense(ds, r)
    return ds, res


def _run(ds, r, prec, path):
    l, n = ds.XL.shape
    m, t = ds.XR.shape[0] // r, ds.Y.shape[0]
    eng = E.Engine(n, l, r, t, m, precision=prec, store_all=True, min_t_store=1.6, min_r2_store=1e-6)
    eng.set_tuning(stats_path=path)
    eng.set_covariates(ds.XL)
    eng.set_traits(ds.Y)
    eng.enable_dense(True)
    eng.run(ds.XR)
    out = eng.dense(m), eng.tuning()["stats_path"]
    eng.close()
    return out


@pytest.mark.parametrize("r", [1, 2])
@pytest.mark.parametrize("patterns,prec", [("few", E.PLAIN), ("own", E.PLAIN), ("own", E.MIXED)])
def test_uncentred_columns(patterns, prec, r):
    ds, res = _data(patterns, r)
    D = res.dense
    assert not D.singular.any()
    (b, se, tt, r2), path = _run(ds, r, prec, 0)
    t_ref = np.abs(D.tstat[:, :, res.l:])
    lim = T_REL * t_ref.max(2, keepdims=True) + T_ABS if prec == E.PLAIN else np.full_like(t_ref, 1e-3)
    dt = np.abs(tt - t_ref)
    assert np.all(dt <= lim), f"max |dt| {dt.max():.3g}"
    assert path == (1 if patterns == "few" else 2)
    if patterns == "own":
        for x, y in zip((b, se, tt, r2), _run(ds, r, prec, 2)[0]):
            np.testing.assert_array_equal(x, y)
