"""Plan calls whose input takes each path of the time-major packing: whole and
ragged channel groups, aligned and unaligned rows and base pointers, sample
counts around its blocks and runs, against the oracle's sums."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nchan,pad,shift", [(64, 0, 0), (128, 16, 0), (68, 0, 0), (63, 0, 0), (65, 3, 0), (64, 0, 1),
                                             (64, 2, 2), (1, 0, 0), (200, 1, 3)])
@pytest.mark.parametrize("rows", [0, 4])
def test_packed_input(hella, oracle, nchan, pad, shift, rows):
    import torch

    plan = hella.Plan(nchan, 1e-3, 468.75, -(468.75 - 375.0) / nchan)
    plan.generate_dm_list(0.0, 25.0, 40.0, 1.25)
    plan.set_pair_rows(rows)
    rng = np.random.default_rng(nchan + pad)
    stride = nchan + pad
    for nout in (1, 200, 257, 1021, 2816, 9000):
        n = plan.max_delay + nout
        x = rng.integers(0, 256, (n, stride), dtype=np.uint8)
        buf = torch.zeros(n * stride + 8, dtype=torch.uint8, device="cuda")
        buf[shift: shift + n * stride] = torch.from_numpy(x.reshape(-1)).cuda()
        out = torch.empty((plan.dm_count, nout), device="cuda")
        torch.cuda.synchronize()
        plan.execute_adv(n, buf.data_ptr() + shift, stride, out, nout * 4, hella.HDD_DEVICE_POINTERS)
        want = oracle.dedisperse(np.ascontiguousarray(x[:, :nchan]), plan.delay_table())
        assert np.array_equal(out.cpu().numpy(), want), nout
