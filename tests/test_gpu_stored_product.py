"""Edges of the stored-product path and of the column-statistics kernel's
layouts: column counts either side of every tile width, ragged columns at
every offset, row sets of every block size, the FP32 screening at high
thresholds, both ways rows come back, scaled inputs of the FP16 split.

Bars: the plain form's against the FP64 oracle (|dt| <= 1e-4 |t| + 1e-4, an
FP32 normal-equation solver's), 1e-3 absolute for the mixed form; paths that
evaluate the same sums in the same order give the same bits.
"""
import numpy as np
import pytest

import quirk_cases as QC
from omicabelnomm_b200 import engine as E
from omicabelnomm_b200 import synth
from test_gpu_parity import T_ABS, T_REL, _yzero, engine_run, oracle_dense

pytestmark = pytest.mark.gpu


def check_plain(ds, r, dense):
    res, _, _ = oracle_dense(ds, r)
    D = res.dense
    ok = ~D.singular
    b, se, tt, r2 = dense
    t_ref = D.tstat[:, :, res.l:][ok]
    dt = np.abs(tt[ok] - t_ref)
    lim = T_REL * np.abs(t_ref) + T_ABS
    assert np.all(dt <= lim), f"max |dt| {dt.max():.3g}, worst ratio {(dt / lim).max():.3g}"
    np.testing.assert_allclose(se[ok], D.se[:, :, res.l:][ok], rtol=1e-4, atol=0)
    np.testing.assert_array_equal(np.isnan(tt[..., 0]), D.singular)
    return res


# (traits, patterns): product columns t + l (1 + patterns) with l = 4 at 63, 64, 65, 127..129, 255..257,
# 288, 300 and the store kernels' narrow / pair boundary
@pytest.mark.parametrize("t,patterns", [(1, 1), (51, 2), (52, 2), (53, 2), (103, 5), (104, 5), (105, 5), (219, 8),
                                        (220, 8), (221, 8), (252, 8), (517, 3)])
def test_plain_product_column_counts(t, patterns):
    ds = synth.generate(synth.scaled(0, n=321, m=259, t=t, l=4, miss_mode="patterns", n_patterns=patterns,
                                     seed=300 + t))
    _, rows, dense = engine_run(ds, 1)
    check_plain(ds, 1, dense)
    assert rows.tests == t * 259


@pytest.mark.parametrize("m", [1, 127, 128, 129, 255, 257])
@pytest.mark.parametrize("r", [1, 2, 4, 8])
def test_plain_product_row_edges(m, r):
    ds = QC.multicol(r, 310 + r, n=260, m=m, t=70, n_patterns=9) if r > 2 else synth.generate(
        synth.scaled(0, n=260, m=m, t=70, l=4, r=r, miss_mode="patterns", n_patterns=9, seed=310 + r))
    _, _, dense = engine_run(ds, r)
    check_plain(ds, r, dense)


@pytest.mark.parametrize("n", [64, 65, 127, 191])
def test_plain_product_short_columns(n):
    """One to three K-blocks, with and without a zero tail."""
    ds = synth.generate(synth.scaled(0, n=n, m=140, t=33, seed=320 + n, miss_frac=0.04))
    _, _, dense = engine_run(ds, 1)
    check_plain(ds, 1, dense)


@pytest.mark.parametrize("xs,ys", [(1e-6, 1e6), (3e4, 1e-5), (7.0, 1e-12)])
def test_plain_product_scaled_inputs(xs, ys):
    """The FP16 split scales every column by a power of two: neither small nor large units lose digits."""
    ds = synth.generate(synth.scaled(0, n=500, m=150, t=40, l=4, miss_mode="patterns", n_patterns=3, seed=331))
    ds.XR[3, 11] = np.float32(400.0)            # an outlier among ordinary values
    # t does not depend on the units; the oracle's own rank rule does, so it sees the unscaled data
    res, _, _ = oracle_dense(ds, 1)
    ok = ~res.dense.singular
    t_ref = res.dense.tstat[:, :, res.l:][ok]
    ds.XR = (ds.XR * np.float32(xs)).astype(np.float32)
    ds.XR[7] *= np.float32(1e-3)
    ds.Y = (ds.Y * np.float32(ys)).astype(np.float32)
    _, _, (_, _, tt, _) = engine_run(ds, 1)
    dt = np.abs(tt[ok] - t_ref)
    lim = T_REL * np.abs(t_ref) + T_ABS
    assert np.all(dt <= lim), f"max |dt| {dt.max():.3g}, worst ratio {(dt / lim).max():.3g}"


@pytest.mark.parametrize("prec", [E.PLAIN, E.MIXED])
@pytest.mark.parametrize("r", [1, 2])
def test_unaligned_columns_give_the_aligned_bits(prec, r):
    """The same SNP block at device offsets of 0 to 3 floats (16-byte aligned copies, copies between the
    boundaries around a column, element copies of the block's edge columns), NaN dosages included."""
    import torch
    for n in (515, 516, 518):
        ds = synth.generate(synth.scaled(0, n=n, m=131, t=20, l=5, r=r, miss_mode="patterns", n_patterns=4,
                                         xr_nan_frac=0.002, seed=340 + n))
        m, t = ds.XR.shape[0] // r, 20
        buf = torch.zeros(ds.XR.size + 8, device="cuda")
        got = []
        for off in range(4):
            buf.fill_(float("inf"))               # whatever surrounds the block must not matter
            buf[off:off + ds.XR.size] = torch.from_numpy(ds.XR.reshape(-1)).cuda()
            eng = E.Engine(n, 5, r, t, m, precision=prec, store_all=True, min_t_store=1.6, min_r2_store=1e-6)
            eng.set_covariates(ds.XL)
            eng.set_traits(ds.Y)
            eng.enable_dense(True)
            torch.cuda.synchronize()
            eng.run_device(buf.data_ptr() + 4 * off, m)
            got.append(eng.dense(m))
            eng.close()
        for d in got[1:]:
            for a, b in zip(got[0], d):
                np.testing.assert_array_equal(a, b)
        if prec == E.PLAIN:
            check_plain(ds, r, got[0])


@pytest.mark.parametrize("r", [1, 2])
@pytest.mark.parametrize("sizes", [(0, 1, 2, 31, 32, 33), (255, 256, 257, 511, 513), (700,) * 45, (700,) * 90])
def test_row_set_sizes(sizes, r):
    """Row sets around the index blocks' sizes; many large sets take work items of two and four blocks."""
    n, t = 1400, len(sizes)
    ds = synth.generate(synth.scaled(0, n=n, m=37, t=t, l=3, r=r, miss_mode="none", seed=350 + len(sizes)))
    rng = np.random.Generator(np.random.PCG64(len(sizes)))
    for j, k in enumerate(sizes):
        ds.Y[j, rng.choice(n, k, replace=False)] = np.nan
    _, _, dense = engine_run(ds, r)
    check_plain(ds, r, dense)


@pytest.mark.parametrize("prec", [E.PLAIN, E.MIXED])
@pytest.mark.parametrize("t,r", [(300, 1), (40, 1), (300, 2), (24, 2)])
def test_screened_rows_are_the_dense_rows(prec, t, r):
    """At |t| > 2.6 and above tests are screened in FP32 first; the stored rows must be exactly those of the
    dense outputs, which every test evaluates in full."""
    min_t = 2.61
    ds = synth.generate(synth.scaled(0, n=700, m=400, t=t, l=4, r=r, effect=0.3, miss_mode="patterns",
                                     n_patterns=5, seed=360 + t))
    m = 400
    out = []
    for dense in (False, True):
        eng = E.Engine(700, 4, r, t, m, precision=prec, min_t_store=min_t, min_r2_store=1e-6)
        eng.set_covariates(ds.XL)
        eng.set_traits(ds.Y)
        eng.enable_dense(dense)
        out.append(eng.run(ds.XR))
        if dense:
            _, _, tt, r2 = eng.dense(m)
        eng.close()
    keep = (tt > np.float32(min_t)).any(2) & (r2 > np.float32(1e-6))
    want = np.argwhere(keep)
    assert len(want) > 50
    for rows in out:
        np.testing.assert_array_equal(np.stack([rows.trait, rows.snp], 1), want)
        np.testing.assert_array_equal(rows.T[:, 4:], tt[keep])
        np.testing.assert_array_equal(rows.r2, r2[keep])


@pytest.mark.parametrize("t,m", [(64, 4095), (64, 4096), (64, 4097), (3, 5)])
def test_rows_come_back_whole(t, m):
    """Around 2^18 stored rows: below in one copy, above in pieces converted by several threads."""
    ds = synth.generate(synth.scaled(0, n=200, m=m, t=t, seed=370 + m))
    _, rows, (b, se, tt, r2) = engine_run(ds, 1)
    ok = ~np.isnan(tt[..., 0])
    want = np.argwhere(ok)
    np.testing.assert_array_equal(np.stack([rows.trait, rows.snp], 1), want)
    l = ds.XL.shape[0]
    for got, dense in ((rows.B, b), (rows.SE, se), (rows.T, tt)):
        np.testing.assert_array_equal(got[:, l:], dense[ok])
    np.testing.assert_array_equal(rows.r2, r2[ok])


@pytest.mark.parametrize("prec", [E.PLAIN, E.MIXED])
@pytest.mark.parametrize("r", [1, 2])
def test_own_patterns_take_the_pre_gemm_within_the_bars(prec, r, monkeypatch):
    """Every trait its own pattern (with zero sets): the pre-GEMM path by default, the row gathers by request."""
    ds = _yzero(synth.generate(synth.scaled(0, n=450, m=90, t=70, l=5, r=r, miss_frac=0.06, seed=380 + r)), 3)
    res, _, _ = oracle_dense(ds, r)
    D = res.dense
    ok = ~D.singular
    t_ref = D.tstat[:, :, res.l:][ok]
    for path in ("", "gather"):
        if path:
            monkeypatch.setenv("OA_STATS_PATH", path)
        eng, _, (_, _, tt, _) = engine_run(ds, r, precision=prec)
        assert eng.tuning()["stats_path"] == (2 if path else 1)
        lim = (T_REL * np.abs(t_ref) + T_ABS) if prec == E.PLAIN else np.full_like(t_ref, 1e-3)
        assert np.all(np.abs(tt[ok] - t_ref) <= lim)


@pytest.mark.parametrize("case", ["chunks", "r2", "r4", "no_intercept", "many_covariates", "yzero"])
def test_noalloc_forms_match_oracle(case):
    """The zero-allocation scan in several chunks, with r = 2 and 4, and where it keeps its FP32 form
    (no intercept; more than eight covariates with two columns per SNP)."""
    from test_zz_no_alloc import noalloc_dense
    r = {"r2": 2, "r4": 4, "many_covariates": 2}.get(case, 1)
    if case == "chunks":
        ds = synth.generate(synth.scaled(0, n=1501, m=2777, t=250, l=5, seed=391))
        ds.XR[2000, 5] = np.nan
    elif case == "r4":
        ds = QC.multicol(4, 392, n=402, m=61, t=30)
    elif case == "many_covariates":
        ds = synth.generate(synth.scaled(0, n=403, m=61, t=14, l=10, r=2, seed=393))
    else:
        ds = synth.generate(synth.scaled(0, n=405, m=131, t=14, l=4, r=r, seed=394))
    if case == "no_intercept":
        ds.XL = np.ascontiguousarray(ds.XL[1:])
    if case == "yzero":
        ds = _yzero(ds, 7)
    if case == "chunks":       # the oracle takes the SNPs either side of the chunks' edges
        got = noalloc_dense(ds, 1)
        pick = np.r_[0:40, 240:270, 500:530, 760:790, 1990:2010, 2740:2777]
        ds.XR = np.ascontiguousarray(ds.XR[pick])
        check_plain(ds, 1, tuple(np.ascontiguousarray(a[:, pick]) for a in got))
    else:
        check_plain(ds, r, noalloc_dense(ds, r))


@pytest.mark.parametrize("prec", [E.PLAIN, E.MIXED])
@pytest.mark.parametrize("model", ["additive", "interaction", "three"])
@pytest.mark.parametrize("n", [517, 518, 2051])
def test_model_columns_give_the_direct_columns_bits(n, model, prec):
    """Dosage models, interactions and zero-padded columns formed on the device (aligned columns with a zero
    tail whatever n) against the same columns passed in."""
    ds = synth.generate(synth.scaled(0, n=n, m=99, t=24, l=4, miss_mode="patterns", n_patterns=4, seed=395 + n))
    rng = np.random.Generator(np.random.PCG64(n))
    r = {"additive": 1, "interaction": 2, "three": 3}[model]
    if model == "additive":
        P = rng.random((99, 3, n)).astype(np.float32)
        raw = P.reshape(297, n)
        direct = np.float32(2.0) * P[:, 0] + P[:, 1]         # 2 x is exact: one rounding, as the fused product
    elif model == "interaction":
        raw = ds.XR
        direct = np.stack([ds.XR * ds.XL[1], ds.XR], 1).reshape(198, n)
    else:
        raw = direct = ds.XR
    out = []
    for cols, formed in ((raw, True), (direct, False)):
        m = cols.shape[0] // (r if model == "three" or not formed else cols.shape[0] // 99)
        eng = E.Engine(n, 4, r, 24, m, precision=prec, store_all=True, min_t_store=1.6, min_r2_store=1e-6)
        eng.set_covariates(ds.XL)
        eng.set_traits(ds.Y)
        if formed and model == "additive":
            eng.set_column_model(3, [2.0, 1.0, 0.0])
        elif formed and model == "interaction":
            eng.set_interactions(ds.XL[1:2])
        eng.enable_dense(True)
        eng.run(np.ascontiguousarray(cols))
        out.append(eng.dense(m))
        eng.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("prec", [E.PLAIN, E.MIXED])
@pytest.mark.parametrize("l,r", [(3, 1), (4, 2), (8, 1), (9, 1), (5, 2)])
def test_many_systems_per_thread_give_the_same_bits(l, r, prec):
    """Schur systems taken eight row sets a thread (12,500 SNPs x 201 slots) against the same SNPs in a block
    small enough for one a thread, covariates in 4, 8 and 16 registers."""
    n, m, t, few = 120, 12500, 200, 67
    ds = synth.generate(synth.scaled(0, n=n, m=m, t=t, l=l, r=r, miss_frac=0.05, seed=400 + l))
    out = []
    for mb in (m, few):
        eng = E.Engine(n, l, r, t, mb, precision=prec, min_t_store=8.0, min_r2_store=1e-6)
        eng.set_tuning(chunk_snps=m)
        eng.set_covariates(ds.XL)
        eng.set_traits(ds.Y)
        eng.enable_dense(True)
        eng.run(np.ascontiguousarray(ds.XR[:mb * r]))
        assert eng.tuning()["stats_path"] == 1
        out.append(eng.dense(mb))
        eng.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a[:, :few], b)


def test_plain_product_in_trait_segments():
    """More traits than one stored product holds (8,192): the last segment and its edges."""
    t = 8192 + 131
    ds = synth.generate(synth.scaled(0, n=130, m=40, t=t, l=3, miss_mode="patterns", n_patterns=3, seed=411))
    _, rows, dense = engine_run(ds, 1)
    check_plain(ds, 1, dense)
    assert rows.tests == 40 * t


@pytest.mark.parametrize("prec", [E.PLAIN, E.MIXED])
def test_statistics_path_changed_after_the_traits(prec):
    """The pre-GEMM's columns are added behind a trait block that was set while the row gathers were chosen."""
    ds = synth.generate(synth.scaled(0, n=333, m=140, t=60, l=4, miss_mode="patterns", n_patterns=7, seed=412))
    out = []
    for late in (False, True):
        eng = E.Engine(333, 4, 1, 60, 140, precision=prec, store_all=True, min_t_store=1.6, min_r2_store=1e-6)
        eng.set_tuning(stats_path=2 if late else 1)
        eng.set_covariates(ds.XL)
        eng.set_traits(ds.Y)
        eng.set_tuning(stats_path=1)
        eng.enable_dense(True)
        eng.run(ds.XR)
        out.append(eng.dense(140))
        eng.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("n,r", [(9599, 2), (9600, 2), (9601, 2), (16384, 1), (12800, 4)])
def test_long_columns(n, r):
    """Either side of the lengths from which a SNP's columns take a group of 512 threads."""
    ds = QC.multicol(r, 420, n=n, m=19, t=6, n_patterns=2) if r > 2 else synth.generate(
        synth.scaled(0, n=n, m=19, t=6, l=4, r=r, miss_mode="patterns", n_patterns=2, seed=420))
    _, _, dense = engine_run(ds, r)
    check_plain(ds, r, dense)


def test_few_and_many_rows_with_covariate_terms():
    """Rows with every covariate term: one block whose rows come back in pieces against two that are formed on
    the device as the caller gets them."""
    t, m = 64, 4099
    ds = synth.generate(synth.scaled(0, n=150, m=m, t=t, l=5, miss_mode="patterns", n_patterns=4, seed=430))
    _, whole, _ = engine_run(ds, 1, disp_cov=True)
    assert len(whole.trait) > 1 << 18
    half = []
    for lo, hi in ((0, 2050), (2050, m)):
        part = type(ds)(**{**ds.__dict__, "XR": np.ascontiguousarray(ds.XR[lo:hi])})
        _, rows, _ = engine_run(part, 1, disp_cov=True)
        assert len(rows.trait) <= 1 << 18
        half.append((rows, lo))
    key = np.concatenate([rows.trait.astype(np.int64) * m + rows.snp + lo for rows, lo in half])
    order = np.argsort(key)
    np.testing.assert_array_equal(key[order], whole.trait.astype(np.int64) * m + whole.snp)
    for field in ("r2", "mask", "B", "SE", "T"):
        got = np.concatenate([getattr(rows, field) for rows, _ in half])[order]
        np.testing.assert_array_equal(got, getattr(whole, field))
