"""The flagger's passes at the edges of their tiles (channel slices and chunks,
warps and rounds of blocks, short chains), bit for bit against the oracle."""
import numpy as np
import pytest

from helpers import small_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nchan,gulp", [(32, 256), (64, 288), (96, 544), (128, 256), (160, 2080), (224, 1024),
                                        (96, 4896), (2048, 512), (8192, 256), (32, 77856)])
def test_flagger_edges(hella, oracle, nchan, gulp):
    rng = np.random.default_rng(nchan + gulp)
    x = np.clip(rng.normal(120, 25, (gulp, nchan)) + np.linspace(0, 60, nchan), 0, 255).astype(np.uint8)
    x[:, 1] = 0
    x[:, 2] = 255
    x[:, 3] = rng.integers(0, 256, gulp)
    x[gulp // 3] = 255  # samples above and below all others
    x[gulp // 2] = 0
    s = hella.Search(hella.default_params(**small_params(nchan=nchan, gulp=gulp, df_mhz=-(468.75 - 375.0) / nchan,
                                                         dm_max=20.0)))
    s.load_gulp(x[None])
    s.fast_flagger()
    out, ts, tr = oracle.flag_beam(x)
    st = s.flag_stats(0)

    def same(a, b):  # bit for bit; which NaN an operation makes is not defined
        a, b = np.float32(a), np.float32(b)
        return np.array_equal(np.where(np.isnan(a), 0, a.view(np.uint32)), np.where(np.isnan(b), 0, b.view(np.uint32)))

    for k in ("bp1", "bp2", "bp3", "mean1", "std1", "mean2", "std2"):
        assert same(st[k], tr[k]), k
    assert same(st["ts"], ts)
    if not np.isnan(st["mean2"]):  # the byte of a NaN is not defined either
        assert np.array_equal(s.copy_window(0)[-gulp:], out)
