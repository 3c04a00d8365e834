"""Group rows at the edges of their build and sum: output lengths around half a
tile, a tile and a build chunk, rings shorter than a chunk's window (several
copies a channel), last groups of one to three channels, against the oracle's
sums."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("channels", [2, 4])
@pytest.mark.parametrize("nchan", [64, 65, 66, 67, 5])
@pytest.mark.parametrize("dm_max", [3.0, 150.0])
def test_rows_at_chunk_edges(hella, oracle, channels, nchan, dm_max):
    plan = hella.Plan(nchan, 1e-3, 468.75, -(468.75 - 375.0) / nchan)
    plan.generate_dm_list(0.0, dm_max, 40.0, 1.25)
    plan.set_pair_rows(channels)
    rng = np.random.default_rng(nchan)
    for nout in (1, 255, 256, 257, 513, 1024, 1025, 2047, 2304, 4097, 6200):
        x = rng.integers(0, 256, (plan.max_delay + nout, nchan), dtype=np.uint8)
        x[: nout // 2 + 1] = 255  # the largest sums a lane holds
        assert np.array_equal(plan.dedisperse(x), oracle.dedisperse(x, plan.delay_table())), nout


@pytest.mark.parametrize("channels,nchan", [(4, 1024), (2, 1024), (4, 261), (2, 515)])
def test_rows_at_the_largest_sums(hella, oracle, channels, nchan):
    """All samples 255 over more channels than the 16-bit lanes hold at once."""
    plan = hella.Plan(nchan, 1e-3, 468.75, -(468.75 - 375.0) / nchan)
    plan.generate_dm_list(0.0, 12.0, 40.0, 1.25)
    plan.set_pair_rows(channels)
    x = np.full((plan.max_delay + 1700, nchan), 255, np.uint8)
    x[::7, ::3] = 1
    assert np.array_equal(plan.dedisperse(x), oracle.dedisperse(x, plan.delay_table()))


@pytest.mark.parametrize("channels,limit", [(2, 43008), (4, 14336)])
@pytest.mark.parametrize("nchan", [16, 19])
def test_rows_at_the_widest_delay_range(hella, oracle, channels, limit, nchan):
    """Group rows up to the largest range of relative delays that the build's
    shared memory holds; the next DM goes channel by channel."""
    plan = hella.Plan(nchan, 65.5e-6, 468.75, -(468.75 - 375.0) / nchan)
    plan.set_pair_rows(channels)

    def span(dm):
        plan.set_dm_list(np.float32([0.0, 0.37 * dm, dm]))
        return plan.pair_tables(0, 3, channels, 8, 2)["max_span"]

    lo, hi = 1.0, 2.0e4
    while hi - lo > 1e-3 * lo / limit:
        mid = (lo + hi) / 2
        lo, hi = (mid, hi) if span(mid) <= limit else (lo, mid)
    rng = np.random.default_rng(channels)
    for dm, kernels in ((lo, 3), (hi, 2)):  # packing, build and sums; packing and sums
        assert (span(dm) <= limit) == (kernels == 3) and abs(span(dm) - limit) <= 1
        x = rng.integers(0, 256, (plan.max_delay + 1500, nchan), dtype=np.uint8)
        before = hella.kernel_launches()
        got = plan.dedisperse(x)
        assert hella.kernel_launches() - before == kernels
        assert np.array_equal(got, oracle.dedisperse(x, plan.delay_table(), nout=1500))
