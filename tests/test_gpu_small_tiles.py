"""Channel-by-channel dedispersion with the tile size chosen by the number of
work items (16 down to 4 trials), on samples of 255 among others (byte lanes as
full as they get), against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nchan", [1, 9, 128, 600])
@pytest.mark.parametrize("ndm", [1, 3, 17, 143, 1300])
def test_tiles_by_item_count(hella, oracle, nchan, ndm):
    plan = hella.Plan(nchan, 1e-3, 468.75, -(468.75 - 375.0) / nchan)
    plan.set_dm_list(np.linspace(0.0, 40.0, ndm, dtype=np.float32))
    rng = np.random.default_rng(ndm)
    for nout in (1, 255, 1024, 1025, 5000):
        x = rng.integers(0, 256, (plan.max_delay + nout, nchan), dtype=np.uint8)
        x[nout // 3: nout // 3 + 300] = 255
        assert np.array_equal(plan.dedisperse(x), oracle.dedisperse(x, plan.delay_table())), nout

