"""Device memory of an engine: what a trait block holds, and blocks near the
end of the memory."""
import numpy as np
import pytest

from omicabelnomm_b200 import engine as E
from omicabelnomm_b200 import synth

pytestmark = pytest.mark.gpu


def _block(n=20000, t=64, l=3, patterns=5):
    ds = synth.generate(synth.scaled(0, n=n, m=8, t=t, l=l, miss_mode="patterns", n_patterns=patterns, seed=800))
    # columns [Y~ | Q | Q o m_1 | ...] in 16-bit hi and lo, and tables of a few rows per pattern and covariate
    n_pad = (n + 63) // 64 * 64
    return ds, 4 * n_pad, (t + l * (1 + patterns)) * 4 * n_pad


@pytest.mark.parametrize("prec", [E.PLAIN, E.MIXED])
def test_trait_block_holds_its_columns_once(prec):
    import torch
    ds, column, columns = _block()
    l, n = ds.XL.shape
    y = torch.from_numpy(ds.Y).cuda()
    torch.cuda.synchronize()
    eng = E.Engine(n, l, 1, 64, 1000, precision=prec, min_t_store=5.0, min_r2_store=1e-6)
    eng.set_covariates(ds.XL)
    before = eng.device_bytes()
    eng.set_traits_device(y.data_ptr(), 64)
    held = eng.device_bytes() - before
    assert columns <= held < columns + 16 * column, (held / column, columns / column)
    eng.close()


class _Rest:
    """Leaves `left` bytes of the GPU's memory free while it is held."""

    def __init__(self, left):
        import torch
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        self.hog = torch.empty(free - left, dtype=torch.uint8, device="cuda") if free > left else None

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        import torch
        self.hog = None
        torch.cuda.empty_cache()


def _scan(XL, Y, X, m, left, prec, **tuning):
    """(dense results, tuning in effect) of an engine that may use `left` bytes (None: all there is)."""
    import torch
    l, n = XL.shape
    eng = E.Engine(n, l, 1, Y.shape[0], m, precision=prec, min_t_store=4.0, min_r2_store=1e-6)
    try:
        eng.set_tuning(**tuning)
        eng.set_covariates(XL)
        with _Rest(left) if left else torch.no_grad():
            eng.set_traits_device(Y.data_ptr(), Y.shape[0])
            eng.enable_dense(True)
            rows = [eng.scan(X.data_ptr(), m) for _ in range(3)]      # the third from the graph
            out = eng.dense(m)
            got = eng.tuning()
    finally:
        eng.close()      # its memory pool goes back to the device
    for r in rows[1:]:
        np.testing.assert_array_equal(rows[0].T, r.T)
    return out, got


@pytest.mark.parametrize("prec", [E.PLAIN, E.MIXED])
def test_chunk_follows_the_memory_that_is_left(prec):
    """A chunk's buffers (1.6 GB at n = 25,000) that do not fit: fewer SNPs per chunk, the same bits."""
    import torch
    n, m, t = 25000, 17000, 24
    ds = synth.generate(synth.scaled(0, n=n, m=4, t=t, l=4, miss_mode="patterns", n_patterns=3, seed=810))
    g = torch.Generator(device="cuda").manual_seed(81)
    X = torch.rand((m, n), generator=g, device="cuda").mul_(2.0)
    Y = torch.from_numpy(ds.Y).cuda()
    torch.cuda.synchronize()
    want, auto = _scan(ds.XL, Y, X, m, None, prec)
    got, cut = _scan(ds.XL, Y, X, m, 900 << 20, prec)
    assert 256 <= cut["chunk_snps"] < auto["chunk_snps"]
    for a, b in zip(want, got):
        np.testing.assert_array_equal(a, b)
    with pytest.raises(E.OAError) as err:                          # a chunk that was asked for is not cut
        _scan(ds.XL, Y, X, m, 900 << 20, prec, chunk_snps=m)
    assert err.value.status == 6


def test_wide_block_whose_columns_do_not_fit_takes_the_gathers():
    """300 traits with own patterns and 16 covariates: 4,832 pre-GEMM columns, 387 MB at n = 20,000."""
    import torch
    n, m, t = 20000, 64, 300
    ds = synth.generate(synth.scaled(0, n=n, m=m, t=t, l=16, miss_frac=0.01, seed=811))
    X, Y = torch.from_numpy(ds.XR).cuda(), torch.from_numpy(ds.Y).cuda()
    torch.cuda.synchronize()
    _, auto = _scan(ds.XL, Y, X, m, None, E.PLAIN)
    want, forced = _scan(ds.XL, Y, X, m, None, E.PLAIN, stats_path=2)
    got, cut = _scan(ds.XL, Y, X, m, 256 << 20, E.PLAIN)
    assert (auto["stats_path"], forced["stats_path"], cut["stats_path"]) == (1, 2, 2)
    for a, b in zip(want, got):
        np.testing.assert_array_equal(a, b)
