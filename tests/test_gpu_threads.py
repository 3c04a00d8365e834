"""Contexts and plans of different sizes used from two threads at once: a
launch's shared memory is its own, whatever the other thread launches of the
same kernel."""
import threading

import numpy as np
import pytest

from helpers import small_params

pytestmark = pytest.mark.gpu

N = 4000  # calls a thread


def _both(jobs):
    errors, gate = [], threading.Barrier(len(jobs))

    def run(job):
        gate.wait()
        try:
            for _ in range(N):
                job()
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=run, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors


def _search(hella, width_max):
    p = small_params(nchan=32, gulp=256, dm_max=5.0, width_max=width_max, df_mhz=-(468.75 - 375.0) / 32)
    s = hella.Search(hella.default_params(**p))
    x = np.random.default_rng(0).integers(100, 156, (1, 256, 32), dtype=np.uint8)
    for _ in range(s.info.min_gulp + 1):
        s.process_gulp(x)
    s.load_gulp(x)
    s.fast_flagger()
    s.dedisperse(0)
    return s


def test_smoothing_of_different_widths(hella):
    import torch

    _both([s.smooth for s in (_search(hella, 100), _search(hella, 4096))])
    torch.cuda.synchronize()


@pytest.mark.parametrize("rows", [0, 2])
def test_plans_of_different_ranges(hella, oracle, rows):
    import torch

    jobs, checks = [], []
    for dm in (5.0, 240.0):
        plan = hella.Plan(64, 1e-3, 468.75, -(468.75 - 375.0) / 64)
        plan.set_dm_list(np.linspace(0.0, dm, 48, dtype=np.float32))
        plan.set_pair_rows(rows)
        plan.set_stream(torch.cuda.Stream().cuda_stream)
        x = np.random.default_rng(1).integers(0, 256, (plan.max_delay + 300, 64), dtype=np.uint8)
        dx, out = torch.from_numpy(x).cuda(), torch.empty((48, 300), device="cuda")
        torch.cuda.synchronize()
        jobs.append(lambda plan=plan, dx=dx, out=out: plan.execute_adv(
            dx.shape[0], dx, 64, out, 300 * 4, hella.HDD_DEVICE_POINTERS | hella.HDD_ASYNC))
        checks.append((out, oracle.dedisperse(x, plan.delay_table(), nout=300)))
    for j in jobs:
        j()
    before = hella.kernel_launches()
    _both(jobs)
    torch.cuda.synchronize()
    assert hella.kernel_launches() - before == 2 * N * (3 if rows else 2)  # none refused, none on another route
    for out, want in checks:
        assert np.array_equal(out.cpu().numpy(), want)
