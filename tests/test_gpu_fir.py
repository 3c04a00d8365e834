"""Smoothing planes and per-width statistics bit for bit against the oracle at
the edges of the FIR kernels' tiles: gulps that end inside the first 256
outputs' successor, a 1024- or a 2048-output iteration, rows that are not
16-byte aligned (odd wmax), widths of one iteration's halo and more, width
lists that split between the two kernels."""
import numpy as np
import pytest

from helpers import small_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gulp", [256, 1024, 1056, 2080, 3072, 4128])
@pytest.mark.parametrize("wmin,wmax", [(1, 2), (1, 33), (1, 64), (1, 100), (1, 512), (3, 50), (2, 64), (7, 4096),
                                       (1025, 2000)])
@pytest.mark.parametrize("anchor", [0, 1])
def test_planes_at_tile_edges(hella, oracle, gulp, wmin, wmax, anchor):
    p = small_params(nchan=64, gulp=gulp, dm_max=30.0, width_min=wmin, width_max=wmax, smooth_anchor=anchor)
    p["df_mhz"] = -(468.75 - 375.0) / 64
    s = hella.Search(hella.default_params(**p))
    rng = np.random.default_rng(gulp + wmax)
    for _ in range(s.info.min_gulp):
        s.process_gulp(rng.integers(100, 156, (1, gulp, 64), dtype=np.uint8))
    s.load_gulp(rng.integers(100, 156, (1, gulp, 64), dtype=np.uint8))
    s.fast_flagger()
    s.dedisperse(0)
    s.smooth(1)
    want, wmean, wstd = oracle.smooth_normalise(s.copy_dedisp(), wmin, wmax, gulp, anchor)[:3]
    mean, std, _ = s.smooth_stats()
    assert np.array_equal(mean.view(np.uint32), wmean.view(np.uint32))
    assert np.array_equal(std.view(np.uint32), wstd.view(np.uint32))
    assert np.array_equal(s.copy_boxes().view(np.uint32), want.view(np.uint32))
