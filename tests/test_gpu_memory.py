"""Device memory of an engine: what a trait block holds, and what oa_reserve
leaves to be allocated."""
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


@pytest.mark.parametrize("prec", [E.PLAIN, E.MIXED])
def test_reserved_engine_takes_a_trait_block_without_growing(prec):
    import torch
    ds, column, columns = _block()
    l, n = ds.XL.shape
    y = torch.from_numpy(ds.Y).cuda()
    torch.cuda.synchronize()
    eng = E.Engine(n, l, 1, 64, 1000, precision=prec, min_t_store=5.0, min_r2_store=1e-6)
    eng.set_covariates(ds.XL)
    eng.reserve(64, 1000)
    before = eng.device_bytes()
    eng.set_traits_device(y.data_ptr(), 64)
    grown = eng.device_bytes() - before
    assert grown < 10 * column, grown / column      # the tables of the row sets, no column buffer
    eng.close()
