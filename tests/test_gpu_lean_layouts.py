"""Layouts of the column-statistics kernel: SNPs per group give the same bits,
256 and 512 threads per CTA the oracle's numbers (they sum in another order)."""
import numpy as np
import pytest

import quirk_cases as QC
from omicabelnomm_b200 import engine as E
from omicabelnomm_b200 import synth
from test_gpu_parity import T_ABS, T_REL, engine_run, oracle_dense

pytestmark = pytest.mark.gpu


def _dense(ds, r, prec, spb):
    l, n = ds.XL.shape
    m, t = ds.XR.shape[0] // r, ds.Y.shape[0]
    eng = E.Engine(n, l, r, t, m, precision=prec, store_all=True, min_t_store=1.6, min_r2_store=1e-6)
    eng.set_tuning(lean_spb=spb, stats_path=1)
    eng.set_covariates(ds.XL)
    eng.set_traits(ds.Y)
    eng.enable_dense(True)
    eng.run(ds.XR)
    out = eng.dense(m)
    eng.close()
    return out


# few patterns and every trait its own (the wide blocks' kernels, 4 and 8 covariate slots); one SNP in seven
# far from zero, one with missing dosages
@pytest.mark.parametrize("prec", [E.PLAIN, E.MIXED])
@pytest.mark.parametrize("r,l,own", [(1, 4, False), (1, 4, True), (1, 7, True), (2, 4, False), (2, 4, True)])
def test_snps_per_group_give_the_same_bits(r, l, own, prec):
    ds = synth.generate(synth.scaled(0, n=1003, m=201, t=70, l=l, r=r, seed=820 + r + l,
                                     **({} if own else dict(miss_mode="patterns", n_patterns=5))))
    ds.XR[::7 * r] += np.float32(30.0)
    ds.XR[5::11 * r, 17] = np.nan
    out = [_dense(ds, r, prec, spb) for spb in (1, 2, 4, 8)]
    for d in out[1:]:
        for a, b in zip(out[0], d):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("prec", [E.PLAIN, E.MIXED])
@pytest.mark.parametrize("n,r,own", [(9700, 2, False), (9700, 2, True), (4900, 4, False), (16400, 1, True)])
def test_thread_counts_match_the_oracle(n, r, own, prec, monkeypatch):
    over = {} if own else dict(miss_mode="patterns", n_patterns=3)
    ds = (QC.multicol(r, 830, n=n, m=21, t=70, n_patterns=3) if r > 2 else
          synth.generate(synth.scaled(0, n=n, m=21, t=70, l=4, r=r, seed=830 + r, **over)))
    res, _, _ = oracle_dense(ds, r)
    t_ref = np.abs(res.dense.tstat[:, :, res.l:])
    t_sys = t_ref.max(2, keepdims=True)
    lim = T_REL * t_sys + T_ABS if prec == E.PLAIN else 1e-3 + 1e-4 * t_sys
    for threads in ("512", "256"):
        monkeypatch.setenv("OA_LEAN_THREADS", threads)
        _, _, dense = engine_run(ds, r, precision=prec)
        dt = np.abs(dense[2] - t_ref)
        assert np.all(dt <= lim), f"{threads} threads: max |dt| {dt.max():.3g}"
