"""The u_tau solves without statistics against the counted ones over the whole
range of y+: the same FP64 root to a relative step of 1e-8, so the same float."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 2_000_000


@pytest.fixture(scope="module")
def wn(built_lib):
    from foil_cfd_gb300 import wallnet
    return wallnet


@pytest.fixture(scope="module")
def torch():
    import torch
    assert torch.cuda.is_available()
    return torch


def samples(wn, torch, lo, hi, seed):
    return [torch.from_numpy(x).cuda() for x in wn.synthetic_samples(N, seed, yplus=(lo, hi))]


@pytest.fixture(scope="module")
def net(wn, torch):
    ut, ys, nu = samples(wn, torch, 1.0, 1e4, 1)
    net = wn.WallNet()
    tau, _ = wn.utau_solve(wn.NEWTON64, ut, ys, nu)
    net.fit_norm(ut, ys, nu, tau)
    return net


@pytest.mark.parametrize("lo,hi", [(1e-7, 1e-5), (1e-5, 1e-3), (1e-3, 9e-3), (9e-3, 0.1), (0.1, 10.0), (10.0, 1e3), (1e3, 1e6)])
@pytest.mark.parametrize("method", ["NEWTON64", "LEARNED", "NEWTON64_NET"])
def test_with_and_without_statistics(wn, torch, net, method, lo, hi):
    m = getattr(wn, method)
    ut, ys, nu = samples(wn, torch, lo, hi, 3)
    a, _ = wn.utau_solve(m, ut, ys, nu, net=net, stats=False)
    b, _ = wn.utau_solve(m, ut, ys, nu, net=net, stats=True)
    apart = (a.view(torch.int32).long() - b.view(torch.int32).long()).abs()
    # Where the short way is taken the root is off by at most the slope's 4e-5
    # times 1e-8: at most one float, and in less than 1e-5 of the samples.
    assert int(apart.max()) <= 1
    assert int((apart > 0).sum()) <= (0 if hi < 0.01 else N // 100_000)
    # The root itself, against Reichardt's law in FP64: at a relative error e of
    # u_tau the residual is at most 2 e (u u+ grows no faster than u^2).
    u = a.double().cpu().numpy()
    up = wn.reichardt_uplus(ys.double().cpu().numpy() * u / nu.double().cpu().numpy())
    if method != "LEARNED" and lo >= 1e-3:
        assert np.max(np.abs(u * up / ut.double().cpu().numpy() - 1)) <= 2 * 2 ** -24 + 1e-8
