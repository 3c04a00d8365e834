"""The flagger's passes at the edges of their tiles (channel slices and chunks,
warps and rounds of blocks, short chains), bit for bit against the oracle."""
import numpy as np
import pytest

from helpers import cands_equal, oracle_pipeline, small_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nchan,gulp,nbeam", [(32, 256, 1), (64, 288, 1), (96, 544, 1), (128, 256, 1), (160, 2080, 1),
                                              (224, 1024, 1), (96, 4896, 1), (1024, 512, 1), (2048, 512, 1),
                                              (8192, 256, 2), (32, 77856, 2)])
def test_flagger_edges(hella, oracle, nchan, gulp, nbeam):
    rng = np.random.default_rng(nchan + gulp)
    x = np.clip(rng.normal(120, 25, (gulp, nchan)) + np.linspace(0, 60, nchan), 0, 255).astype(np.uint8)
    x[:, 1] = 0
    x[:, 2] = 255
    x[:, 3] = rng.integers(0, 256, gulp)
    x[gulp // 3] = 255  # samples above and below all others
    x[gulp // 2] = 0
    s = hella.Search(hella.default_params(**small_params(nchan=nchan, gulp=gulp, df_mhz=-(468.75 - 375.0) / nchan,
                                                         dm_max=20.0, nbeam=nbeam)))
    s.load_gulp(np.stack([x[::-1]] * (nbeam - 1) + [x]))
    s.fast_flagger()
    out, ts, tr = oracle.flag_beam(x)
    st = s.flag_stats(nbeam - 1)

    def same(a, b):  # bit for bit; which NaN an operation makes is not defined
        a, b = np.float32(a), np.float32(b)
        return np.array_equal(np.where(np.isnan(a), 0, a.view(np.uint32)), np.where(np.isnan(b), 0, b.view(np.uint32)))

    for k in ("bp1", "bp2", "bp3", "mean1", "std1", "mean2", "std2"):
        assert same(st[k], tr[k]), k
    assert same(st["ts"], ts)
    if not np.isnan(st["mean2"]):  # the byte of a NaN is not defined either
        assert np.array_equal(s.copy_window(nbeam - 1)[-gulp:], out)


@pytest.mark.parametrize("gulp", [256, 288, 1056, 2080, 8480])
def test_gulp_loop_odd_gulps(hella, oracle, gulp):
    """Words packed over gulps that are no whole blocks and runs, round the ring: the
    dedispersed planes of each gulp against the oracle's on the same window."""
    p = small_params(nchan=96, gulp=gulp, df_mhz=-(468.75 - 375.0) / 96, dm_max=60.0)
    s = hella.Search(hella.default_params(**p))
    pl = oracle_pipeline(oracle, p)
    rng = np.random.default_rng(gulp)
    for g in range(pl.min_gulp + 3):
        x = rng.integers(100, 156, (1, gulp, 96), dtype=np.uint8)
        _, searched = s.process_gulp(x)
        _, expected = pl.gulp_step(x)
        assert searched == expected
        if searched:
            s.clear_peaks()
            s.load_gulp(x)
            s.fast_flagger()
            s.dedisperse(0)
            assert np.array_equal(s.copy_dedisp(), pl.search_window(s.copy_window(0), 0)["dd"]), g
            break


def test_requant_every_half():
    """The output stage's clamp in half precision and its one rounding toward zero
    against the reference's clamp and truncation, for every half."""
    h = np.arange(65536, dtype=np.uint16).view(np.float16)
    h = h[~np.isnan(h)].astype(np.float32)
    scale = np.float32(255) / np.float32(14)
    ref = np.clip(scale * (h + np.float32(4)), 0, 255).astype(np.uint8)
    held = np.clip(h, np.float32(-4), np.float32(10.0078125)) + np.float32(4)
    assert np.array_equal(np.floor(np.float64(scale) * held).astype(np.int64) & 255, ref)


@pytest.mark.parametrize("gulp,snr,cap", [(544, 2.0, 100000), (544, 2.0, 777), (16416, 3.0, 100000), (16416, 2.0, 5001)])
def test_many_candidates(hella, oracle, gulp, snr, cap):
    """Rows full of candidates, several rounds a row and more rows than a scan takes
    at once; the cap reached within a row."""
    p = small_params(nchan=64, gulp=gulp, df_mhz=-(468.75 - 375.0) / 64, dm_max=60.0, dm_tol=1.05, width_max=64, snr=snr,
                     max_giants=cap, always_find_peaks=1)
    s = hella.Search(hella.default_params(**p))
    pl = oracle_pipeline(oracle, p)
    rng = np.random.default_rng(gulp)
    for g in range(pl.min_gulp + 1):
        x = rng.integers(90, 166, (1, gulp, 64), dtype=np.uint8)
        got, _ = s.process_gulp(x)
        want, _ = pl.gulp_step(x)
        assert cands_equal(got, want)
    assert len(got) == cap or cap == 100000 and len(got) > 1000


@pytest.mark.parametrize("nchan,gulp,box", [(32, 288, (1, 1)), (96, 2080, (5, 3)), (160, 544, (16, 8)), (64, 1056, (2, 31))])
def test_planes_edges(hella, oracle, nchan, gulp, box):
    """The fp16 planes' passes at odd sizes, with and without whole batches of loads,
    against the oracle."""
    rng = np.random.default_rng(nchan + gulp)
    x = np.clip(rng.normal(120, 25, (gulp, nchan)), 0, 255).astype(np.uint8)
    x[gulp // 3:gulp // 3 + 5, 3:9] = 255
    p = small_params(nchan=nchan, gulp=gulp, df_mhz=-(468.75 - 375.0) / nchan, dm_max=20.0)
    entries = [(box[0], box[1], 3.0, 1)]
    s = hella.Search(hella.default_params(**p, scrunches=entries))
    fspec = np.zeros(nchan, np.float32)
    s.load_gulp(x[None])
    s.fast_flagger()
    out, ts, _ = oracle.flag_beam(x, oracle.flag_params(scrunches=entries), fspec)
    assert np.array_equal(s.flag_stats(0)["ts"].view(np.uint32), ts.view(np.uint32))
    assert np.array_equal(s.copy_window(0)[-gulp:], out)
    assert np.array_equal(s.flag_spec().view(np.uint32), fspec.view(np.uint32))


@pytest.mark.parametrize("nchan,gulp", [(64, 288), (160, 800), (128, 4128)])
def test_zero_time_series_in_the_tail(hella, oracle, nchan, gulp):
    """A sample whose time series is exactly 0, past the samples that the means
    are taken over: valid statistics, and quotients that are infinite in the
    output stage.  Levels of 96 and 160 in a checkerboard make every table value
    0 or 2; 64 and 128, made up for in the sample after, make -1 and 1."""
    t0 = 256 * (gulp // 256) + 4
    x = np.where((np.arange(nchan)[None] + np.arange(gulp)[:, None]) % 2 == 0, 96, 160).astype(np.uint8)
    even = np.arange(nchan) % 2 == 0
    x[t0], x[t0 + 1] = np.where(even, 64, 128), np.where(even, 192, 128)
    s = hella.Search(hella.default_params(**small_params(nchan=nchan, gulp=gulp, df_mhz=-(468.75 - 375.0) / nchan,
                                                         dm_max=20.0)))
    s.load_gulp(x[None])
    s.fast_flagger()
    out, ts, tr = oracle.flag_beam(x)
    assert ts[t0] == 0 and tr["mean2"] == 1 and tr["std2"] == 1
    assert np.array_equal(out[t0], np.where(even, 0, 255))
    assert np.array_equal(s.flag_stats(0)["ts"], ts)
    assert np.array_equal(s.copy_window(0)[-gulp:], out)
