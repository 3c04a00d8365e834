"""Plan calls queued one behind another on a non-blocking stream, without a
wait between them: several lengths (each with its own tile size and tables),
trial ranges and a new killmask, against the oracle's sums."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [0, 2, 4])
def test_queued_calls_of_several_lengths(hella, oracle, rows):
    import torch

    nchan, ndm = 96, 495
    plan = hella.Plan(nchan, 1e-3, 468.75, -(468.75 - 375.0) / nchan)
    plan.set_dm_list(np.linspace(0.0, 400.0, ndm, dtype=np.float32))
    plan.set_pair_rows(rows)
    stream = torch.cuda.Stream()  # non-blocking: plain copies do not wait for it
    plan.set_stream(stream.cuda_stream)
    rng = np.random.default_rng(rows)
    x = rng.integers(0, 256, (plan.max_delay + 6200, nchan), dtype=np.uint8)
    dx = torch.from_numpy(x).cuda()
    table = plan.delay_table()
    want = oracle.dedisperse(x, table, nout=6200)
    torch.cuda.synchronize()
    # 7, 4 and 1 time tiles: 16-, 8- and 4-trial tiles of all trials
    calls = [(nout, 0, ndm) for nout in (6200, 4000, 900, 6200, 300, 3500)] * 4
    calls += [(6200, 100, 77), (900, 0, ndm), (2000, 300, 195), (6200, 0, ndm)]
    outs = [torch.full((count, nout), -1.0, device="cuda") for nout, _, count in calls]
    torch.cuda.synchronize()
    for (nout, first, count), out in zip(calls, outs):
        plan.execute_guru(plan.max_delay + nout, dx, nchan, out, nout * 4, first, count,
                          flags=hella.HDD_DEVICE_POINTERS | hella.HDD_ASYNC)
    km = np.ones(nchan, np.int32)
    km[::3] = 0
    plan.set_killmask(km)
    last = torch.full((ndm, 4000), -1.0, device="cuda")
    plan.execute_guru(plan.max_delay + 4000, dx, nchan, last, 4000 * 4, 0, ndm,
                      flags=hella.HDD_DEVICE_POINTERS | hella.HDD_ASYNC)
    torch.cuda.synchronize()
    for (nout, first, count), out in zip(calls, outs):
        assert np.array_equal(out.cpu().numpy(), want[first:first + count, :nout]), (nout, first)
    assert np.array_equal(last.cpu().numpy(), oracle.dedisperse(x, table, killmask=km, nout=4000))
    plan.close()
