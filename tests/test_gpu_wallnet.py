"""GPU tests of the learned u_tau seed (include/foilcfd_wallnet.h): the FP64
Newton label/judge kernel against the CPU oracle, the network's forward and
training gradient against the FP64 numpy oracle, deterministic training, the
trained seed's accuracy and what it gains over the method without it (full
FP64 Newton), the harvest of wall-cell samples, and the learned wall update
inside the solver against the full-Newton update."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def wn(built_lib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from foil_cfd_gb300 import wallnet
    return wallnet


@pytest.fixture(scope="module")
def wo():
    from oracle import wallnet_oracle
    return wallnet_oracle


def cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()


def samples(wn, n, seed, harvest_like=0.5):
    """Synthetic samples: a share with the airfoil tunnels' fixed lattice
    viscosities and sample distances, the rest spanning y+ 1..1e4 broadly."""
    ut, ys, nu = wn.synthetic_samples(n, seed)
    k = int(n * harvest_like)
    if k:
        rng = np.random.default_rng(seed + 1000)
        hu, hy, hn = wn.synthetic_samples(k, seed + 2000, yplus=(1.0, 300.0), log10_nu=(-3.78, -3.48), y=(0.5, 3.0))
        ut[:k], ys[:k], nu[:k] = hu, hy, hn
        perm = rng.permutation(n)
        ut, ys, nu = ut[perm], ys[perm], nu[perm]
    return ut, ys, nu


@pytest.fixture(scope="module")
def trained(wn):
    ut, ys, nu = samples(wn, 300_000, seed=11)
    t = [cuda(a) for a in (ut, ys, nu)]
    tau, _ = wn.utau_solve(wn.NEWTON64, *t, stats=False)
    net, hist = wn.train_wallnet(*t, tau, epochs=400, batch=2048, lr_max=3e-3, seed=3)
    return net, hist


def test_newton64_kernel_matches_oracle(wn, oracle_mod):
    ut, ys, nu = wn.synthetic_samples(50_000, seed=10)
    got, st = wn.utau_solve(wn.NEWTON64, cuda(ut), cuda(ys), cuda(nu))
    ref = oracle_mod.utau_newton_f64(ut, ys, nu)
    assert st["solved"] == 50_000 and st["fallbacks"] == 0 and st["newton_iterations"] > 0
    rel = np.abs(got.cpu().numpy().astype(np.float64) - ref) / ref
    assert rel.max() <= 1.2e-7  # FP64 roots agree to 1e-8; output rounded to FP32


def test_forward_and_gradient_match_oracle(wn, wo):
    ut, ys, nu = samples(wn, 20_000, seed=12)
    t = [cuda(a) for a in (ut, ys, nu)]
    tau, _ = wn.utau_solve(wn.NEWTON64, *t, stats=False)
    net = wn.WallNet(seed=7)
    net.fit_norm(*t, tau)
    for round_ in range(2):
        _, b, norm = net.params()
        seed = net.predict(*t).cpu().numpy().astype(np.float64)
        ref = wo.seed(b, norm, ut, ys, nu)
        assert np.max(np.abs(seed - ref) / ref) <= 2e-5
        loss, g = net.gradient(*t, tau)
        x = wo.inputs(norm, ut, ys, nu)
        tgt = wo.target(norm, ut, tau.cpu().numpy())
        lo, go = wo.loss_and_grad(b, x, tgt)
        assert abs(loss - lo) <= 1e-4 * lo
        assert np.linalg.norm(g - go) <= 1e-4 * np.linalg.norm(go)
        assert np.max(np.abs(g - go)) <= 1e-3 * np.max(np.abs(go))
        # Second round: after a few Adam steps the weights are trained ones.
        net.train(*t, tau, epochs=3, batch=4096, seed=1)


def test_training_is_deterministic(wn):
    ut, ys, nu = samples(wn, 50_000, seed=13)
    t = [cuda(a) for a in (ut, ys, nu)]
    tau, _ = wn.utau_solve(wn.NEWTON64, *t, stats=False)
    outs = []
    for _ in range(2):
        net, hist = wn.train_wallnet(*t, tau, epochs=5, batch=4096, seed=9)
        outs.append((net.params()[0], hist))
    assert np.array_equal(outs[0][0], outs[1][0]) and np.array_equal(outs[0][1], outs[1][1])
    assert outs[0][1][-1] < outs[0][1][0]


def test_learned_seed_accuracy_and_gain(wn, wo, trained):
    net, hist = trained
    assert hist[-1] < 1e-5
    ut, ys, nu = samples(wn, 200_000, seed=14)
    t = [cuda(a) for a in (ut, ys, nu)]
    judge, sj = wn.utau_solve(wn.NEWTON64, *t)
    judge = judge.cpu().numpy().astype(np.float64)
    seed = net.predict(*t).cpu().numpy().astype(np.float64)
    seed_err = np.abs(seed - judge) / judge
    assert np.median(seed_err) <= 2e-3
    learned, sl = wn.utau_solve(wn.LEARNED, *t, net=net)
    err = np.abs(learned.cpu().numpy() - judge) / judge
    assert err.max() <= 1e-4, err.max()
    # Fallbacks come from seeds off by more than ~1.4e-3 at y+ < 10, where
    # Newton's quadratic constant is largest (~0.5).
    assert sl["fallbacks"] <= 0.08 * sl["solved"], sl
    # What the network gains over the method without it. (1) With the
    # learned path's budget of one FP32 correction, the network seed settles
    # (residual <= 1e-6) most cells; the reference seed almost none.
    ok_net = wo.one_correction_residual(seed, ut, ys, nu) <= 1e-6
    ok_ref = wo.one_correction_residual(wo.reference_seed(ut, ys, nu), ut, ys, nu) <= 1e-6
    assert ok_net.mean() >= 0.92 and ok_net.mean() >= ok_ref.mean() + 0.5, (ok_net.mean(), ok_ref.mean())
    assert abs(ok_net.mean() - (1 - sl["fallbacks"] / sl["solved"])) <= 0.01
    # (2) Full FP64 Newton to 1e-8 takes fewer iterations from it.
    _, sn = wn.utau_solve(wn.NEWTON64_NET, *t, net=net)
    assert sn["newton_iterations"] < sj["newton_iterations"], (sj, sn)


@pytest.mark.parametrize("n", [1, 255, 257, 4099])
@pytest.mark.parametrize("method", ["NEWTON64", "LEARNED", "NEWTON64_NET"])
def test_solves_without_statistics_match_the_counted_ones(wn, trained, method, n):
    """The short FP64 solve, with sizes around a block, y+ far outside the trained
    range and numbers that FP32 Newton cannot follow. Both stop at a step of 1e-8,
    so two results round to the same or to neighbouring floats."""
    r = np.random.default_rng(n)
    ut = np.exp(r.uniform(np.log(1e-6), np.log(10.0), n)).astype(np.float32)
    ys = np.exp(r.uniform(np.log(1e-3), np.log(1e3), n)).astype(np.float32)
    nu = np.exp(r.uniform(np.log(1e-9), np.log(1.0), n)).astype(np.float32)
    if n > 1:
        ut[:9] = [0.0, -1.0, 1.0, 1e-30, 1e30, np.inf, np.nan, 1.0, 1e-38]
        ys[:9] = [1.0, 1.0, 1e25, 1.0, 1.0, 1.0, 1.0, 1e-30, 0.5]
        nu[:9] = [1e-3, 1e-3, 1e-25, 1e-3, 1e-3, 1e-3, 1e-3, 1e30, 1e-2]
    t = [cuda(a) for a in (ut, ys, nu)]
    net = None if method == "NEWTON64" else trained[0]
    m = getattr(wn, method)
    kw = {} if net is None else {"net": net}
    want, _ = wn.utau_solve(m, *t, **kw)
    got, st = wn.utau_solve(m, *t, stats=False, **kw)
    np.testing.assert_allclose(got.cpu().numpy(), want.cpu().numpy(), rtol=1.2e-7, atol=0, equal_nan=True)


def _time(fn, reps=5):
    best = float("inf")
    for _ in range(reps):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        fn()
        torch.cuda.synchronize()
        best = min(best, time.perf_counter() - t0)
    return best


def test_learned_solve_is_faster_than_full_newton(wn, trained):
    net, _ = trained
    ut, ys, nu = samples(wn, 2_000_000, seed=15)
    t = [cuda(a) for a in (ut, ys, nu)]
    full = _time(lambda: wn.utau_solve(wn.NEWTON64, *t, stats=False))
    learned = _time(lambda: wn.utau_solve(wn.LEARNED, *t, net=net, stats=False))
    assert full >= 2.0 * learned, (full, learned)


def _tunnel(fc):
    from foil_cfd_gb300.tunnels import airfoil_tunnel
    t = airfoil_tunnel(160, 64, 16, chord=64, aoa=6.0, patch=False)
    s = fc.LBMSolver()
    s.init(t.dims, fc.compute_scaling(1.2, 30.0, 1.48e-5, t.chord_cells, t.u_lat), t.flags, les_cs=0.1)
    s.set_wall_model_enabled(True)
    s.set_startup_ramp_enabled(False)
    s.reset()
    assert s.step_n(150) == 0
    return t, s


def test_harvest_matches_sampled_moments(wn, oracle_mod):
    import foil_cfd_gb300 as fc
    t, s = _tunnel(fc)
    n = s.wall_count(0)
    assert n > 100
    ut = torch.empty(n, device="cuda")
    ys = torch.empty(n, device="cuda")
    assert s.wall_harvest(0, ut.data_ptr(), ys.data_ptr(), n) == n
    wl = fc.build_wall_list(t.dims, t.flags)
    assert len(wl["cell"]) == n
    f = s.export_f32().reshape(19, -1).astype(np.float64)
    cx, cy, cz = oracle_mod.CX, oracle_mod.CY, oracle_mod.CZ
    fs = f[:, wl["sample"]]
    rho = np.maximum(fs.sum(0), 0.05)
    u = np.stack([cx @ fs, cy @ fs, cz @ fs]) / rho
    nrm = np.stack([wl["nx"], wl["ny"], wl["nz"]]).astype(np.float64)
    tang = u - (u * nrm).sum(0) * nrm
    ref = np.sqrt((tang ** 2).sum(0))
    cut = 1e-3 * t.u_lat
    got = ut.cpu().numpy()
    on = ref > cut * 1.001
    assert np.allclose(got[on], ref[on], rtol=1e-4, atol=1e-7)
    assert np.array_equal(ys.cpu().numpy(), wl["ys"])


def test_solver_learned_update_matches_full_newton(wn, trained):
    import foil_cfd_gb300 as fc
    net, _ = trained
    t, s = _tunnel(fc)
    utau0, slip0 = s.export_wall_state(0)
    sc = fc.compute_scaling(1.2, 30.0, 1.48e-5, t.chord_cells, t.u_lat)
    nu, cut = (sc.tau - 0.5) / 3.0, 1e-3 * t.u_lat
    res = {}
    for method in (wn.NEWTON64, wn.LEARNED):
        s.import_wall_state(0, utau0, slip0)
        s.set_wall_solver(method, net if method == wn.LEARNED else None)
        s.wall_update_now(0, nu, cut)
        res[method] = s.export_wall_state(0)
    a, b = res[wn.NEWTON64][0], res[wn.LEARNED][0]
    on = a > 0
    assert on.sum() > 100 and np.array_equal(on, b > 0)
    assert np.max(np.abs(b[on] - a[on]) / a[on]) <= 1e-4
    sa = res[wn.NEWTON64][1].view(np.float16).astype(np.float64)
    sb = res[wn.LEARNED][1].view(np.float16).astype(np.float64)
    assert np.all(np.abs(sa - sb) <= 2e-3 * np.abs(sa) + 1e-6)
    # Timed updates report the solve statistics of the selected method.
    s.set_wall_solver(wn.LEARNED, net)
    ms, st = s.wall_update_timed(0, 3)
    assert ms > 0 and st["solved"] > 100 and st["fallbacks"] <= 0.08 * st["solved"]
    s.set_wall_solver(wn.REFERENCE)
    assert s.step_n(50) == 0
