"""The refinement's support rule and its one-launch Adam fit.

CPU: exp(-u^2/2) in fp32 is exactly 0 from |u| = 14.5 on, so an element
outside mu +- 14.75 sigma adds exactly 0 to the gradient sums.  GPU: the fit,
whose passes read the supports only, against Adam steps on the gradients of
the adjoint call, which reads every element."""
import numpy as np
import pytest

import synth

TS, F0 = 1.048576e-3, 468.75
LR = np.float32([0.5, 0.2, 0.05, 0.05, 0.05])


def test_model_vanishes_outside_the_support():
    u = np.arange(14.5, 40.0, 1e-3).astype(np.float32)
    x = np.float32(-0.72134752) * (u * u)
    # half the smallest fp32 denormal is 2^-150: anything below rounds to 0 (2 ulp of exp2f change nothing)
    assert x.max() < -151.0 and np.all(np.exp2(x.astype(np.float64)).astype(np.float32) == 0)


def _adam(theta, grads):
    """Adam in fp32, each multiply-add rounded once (in 64 bits first: a tie apart)."""
    f = np.float32
    m, v = np.zeros_like(theta), np.zeros_like(theta)
    b1 = b2 = 1.0
    for grad in grads:
        g = grad(theta)
        b1, b2 = b1 * 0.9, b2 * 0.999
        m = (np.float64(f(0.9)) * m + f(0.1) * g).astype(f)
        v = (np.float64(f(0.999)) * v + f(0.001) * (g * g)).astype(f)
        theta = theta - LR * (m / f(1.0 - b1)) / (np.sqrt(v / f(1.0 - b2)) + f(1e-8))
        theta[:, 0] = np.fmax(theta[:, 0], f(0))
        theta[:, 2] = np.fmax(theta[:, 2], f(0.05))
    return theta


# channels: one group, fewer groups than a cluster's warps, more groups than that; widths (ms) whose
# supports take 8, 16, 32 and several times 32 float4 groups and more than the row; bursts at the row's
# ends and outside it; a fit of one step (the pass that reads everything) and of several
@pytest.mark.gpu
@pytest.mark.parametrize("nchan,nsamp", [(16, 128), (176, 640), (1040, 2048)])
@pytest.mark.parametrize("width,t0", [(0.05, 0.5), (1.7, 0.5), (4.4, 0.0), (11.0, 1.0), (20.0, 0.5), (400.0, 0.5),
                                      (3.0, 1.2), (3.0, -0.3)])
@pytest.mark.parametrize("steps", [1, 4])
def test_fit_matches_adam_on_the_adjoint(hella, nchan, nsamp, width, t0, steps):
    import torch

    n, df = 3, -(468.75 - 375.0) / nchan
    rng = np.random.default_rng(nchan + int(width * 10))
    cut = torch.from_numpy(rng.standard_normal((n, nchan, nsamp), dtype=np.float32)).cuda()
    dm_ref = torch.tensor([150.0, 900.0, 1800.0], device="cuda")
    theta0 = np.stack([dm_ref.cpu().numpy() + 0.3, np.full(n, t0 * nsamp), np.full(n, width), np.full(n, 0.8),
                       rng.uniform(-2, 2, n)], 1).astype(np.float32)
    r = hella.Refine(4, nchan, nsamp, TS, F0, df, stream=torch.cuda.current_stream().cuda_stream)
    one, out = torch.ones(n, device="cuda"), torch.empty((n, 5), device="cuda")

    def grad(theta):
        r.adjoint(cut, dm_ref, torch.from_numpy(theta).cuda(), one, out)
        return out.cpu().numpy()

    want = _adam(theta0, [grad] * steps)
    before = _adam(theta0, [grad] * (steps - 1))
    theta, chi2, want_chi2 = torch.from_numpy(theta0).cuda(), torch.empty(n, device="cuda"), torch.empty(n, device="cuda")
    r.fit(cut, dm_ref, theta, steps, LR, chi2)
    r.forward(cut, dm_ref, torch.from_numpy(before).cuda(), want_chi2)
    # the gradients are the same sums in the same order: what is left is a few ulp an Adam step
    assert np.allclose(theta.cpu().numpy(), want, rtol=2e-6, atol=2e-6)
    assert np.allclose(chi2.cpu().numpy(), want_chi2.cpu().numpy(), rtol=2e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("steps", [1, 3])
def test_non_finite_samples_reach_the_results(hella, bad, steps):
    """A non-finite sample far from the burst: its cutout's gradient and fit
    are not finite (dm and width at their floors), the others' are."""
    import torch

    n, nchan, nsamp = 2, 64, 1024
    truth, dm_ref, theta0 = synth.refine_truth(n, np.arange(0.0, 2001.0, 25.0), nchan=nchan, nsamp=nsamp, seed=3)
    cut = torch.randn((n, nchan, nsamp), device="cuda")
    cut[1, 40, 3] = float(bad)
    r = hella.Refine(n, nchan, nsamp, TS, F0, -(468.75 - 375.0) / nchan, stream=torch.cuda.current_stream().cuda_stream)
    dm, theta = torch.from_numpy(dm_ref).cuda(), torch.from_numpy(theta0).cuda()
    out, chi2 = torch.empty((n, 5), device="cuda"), torch.empty(n, device="cuda")
    r.adjoint(cut, dm, theta, torch.ones(n, device="cuda"), out)
    assert torch.isfinite(out[0]).all() and torch.isnan(out[1]).all()
    r.fit(cut, dm, theta, steps, LR, chi2)
    got, c = theta.cpu().numpy(), chi2.cpu().numpy()
    assert np.isfinite(got[0]).all() and np.isfinite(c[0])
    assert got[1, 0] == 0 and got[1, 2] == np.float32(0.05) and np.isnan(got[1, [1, 3, 4]]).all()
    assert not np.isfinite(c[1]) and (steps == 1 or np.isnan(c[1]))


@pytest.mark.gpu
def test_calls_after_overlapping_calls(hella):
    """Calls of one context on two streams without an order between them leave
    their own results undefined, never those of the calls after them."""
    import torch

    n, nchan, nsamp = 24, 1024, 512
    r = hella.Refine(n, nchan, nsamp, TS, F0, -(468.75 - 375.0) / nchan)
    cut = torch.randn((n, nchan, nsamp), device="cuda")
    dm = torch.full((n,), 300.0, device="cuda")
    theta = torch.tensor([300.2, nsamp / 2, 5.0, 0.7, 0.3], device="cuda").repeat(n, 1)
    one = torch.ones(n, device="cuda")
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]

    def calls():
        chi2, grad = torch.full((n,), -1.0, device="cuda"), torch.full((n, 5), -1.0, device="cuda")
        torch.cuda.synchronize()
        r.forward(cut, dm, theta, chi2)
        r.adjoint(cut, dm, theta, one, grad)
        torch.cuda.synchronize()
        return chi2.cpu().numpy(), grad.cpu().numpy()

    chi2, grad = calls()
    for _ in range(5):
        outs = [(torch.empty(n, device="cuda"), torch.empty((n, 5), device="cuda")) for _ in streams]
        torch.cuda.synchronize()
        for _ in range(10):
            for s, (c, g) in zip(streams, outs):
                r.set_stream(s.cuda_stream)
                r.forward(cut, dm, theta, c)
                r.adjoint(cut, dm, theta, one, g)
        torch.cuda.synchronize()
        after = calls()
        assert np.array_equal(after[0], chi2) and np.array_equal(after[1], grad)
