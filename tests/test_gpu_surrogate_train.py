"""Surrogate end to end on the GPU: data from the walk, training on the tensor-core
kernels, what the network gains over plain Monte Carlo, and the Gauss-Newton inverse."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

from monte_carlompi_gb300 import inverse, surrogate  # noqa: E402


@pytest.fixture(scope='module')
def trained(walker):
    ds = surrogate.make_dataset(walker, 1536, 50000, seed=101)
    hold = 96
    train = surrogate.Dataset(ds.x[hold:], ds.y[hold:], ds.raw[hold:], ds.brf[hold:], ds.albedo[hold:],
                              ds.photons)
    ens = surrogate.train(train, members=3, epochs=150, batch=256, lr=1e-3, seed=1)
    return ens, ds, hold


def test_network_beats_the_monte_carlo_it_learned_from(walker, trained):
    """Gain over the method without it: on held-out configs the network, trained on
    5e4-photon walks, is closer to a 2e6-photon walk than a 5e4-photon walk is, and it
    answers in microseconds instead of milliseconds."""
    ens, ds, hold = trained
    judge, _ = surrogate.mc_brf(walker, ds.raw[:hold], 2000000, seed=202)
    pred, _, _ = ens.predict(ds.raw[:hold])
    err_net = surrogate.rel_rms(pred, judge)
    err_mc = surrogate.rel_rms(ds.brf[:hold], judge)
    assert np.median(err_net) < 0.8 * np.median(err_mc), (np.median(err_net), np.median(err_mc))
    assert np.median(err_net) < 0.06
    assert surrogate.inference_rate(ens, batch=16384, reps=5) > 1e6


def test_jacobian_matches_cpu_autograd(trained):
    """d BRF / d log r_eff from the batched autograd pass through the kernels equals
    float64 CPU autograd of the same network (bf16 roundings included)."""
    from tests.helpers import reference_mlp
    ens, ds, _ = trained
    one = surrogate.Ensemble(ens.members[:1])
    m = ens.members[0]
    known = ds.raw[:8, 1:]
    s = np.log(ds.raw[:8, 0])
    f, jac = inverse._brf_and_jacobian(one, s, known)
    params = [p.detach().cpu().double() for p in m.params]
    y_mean, y_std = m.y_mean.cpu().double(), m.y_std.cpu().double()
    lo, hi = inverse.LOG_R

    def brf_of(sv):
        r = torch.exp(sv)
        x = torch.stack([2 * (torch.log(r) - lo) / (hi - lo) - 1,
                         *[torch.from_numpy(surrogate.encode(np.exp(s), known[:, 0], known[:, 1],
                                                             known[:, 2])[:, k]).double()
                           for k in (1, 2, 3)]], dim=1)
        y = reference_mlp(x, params) * y_std + y_mean
        alb = torch.exp(y[:, surrogate.N_BRF])
        return (torch.exp(y[:, :surrogate.N_BRF]) - surrogate.BRF_FLOOR) * alb[:, None]

    sv = torch.from_numpy(s).double().requires_grad_(True)
    ref_f = brf_of(sv)
    ref_j = torch.stack([torch.autograd.grad(ref_f[:, b].sum(), sv, retain_graph=True)[0]
                         for b in range(surrogate.N_BRF)], dim=1).numpy()
    w = surrogate.bin_weights()
    assert np.max(np.abs(f - ref_f.detach().numpy())) < 2e-2 * np.max(np.abs(f))
    rel = np.sqrt(((jac - ref_j) ** 2 * w).sum(1) / ((ref_j ** 2 * w).sum(1) + 1e-30))
    assert np.median(rel) < 0.03, np.median(rel)


def test_gauss_newton_recovers_r_eff_on_network_brfs(trained):
    ens, ds, _ = trained
    rng = np.random.default_rng(7)
    raw = surrogate.sample_inputs(64, 303)
    raw[:, 1] = rng.uniform(1.4, 1.8, 64)          # absorbing wavelengths: r_eff is well constrained
    obs, _, _ = ens.predict(raw)
    s, _, spread, spread_r = inverse.surrogate_gn(ens, obs, raw[:, 1:])
    err = np.abs(np.exp(s) / raw[:, 0] - 1)
    assert np.median(err) < 0.01, np.median(err)
    assert np.all(np.isfinite(s)) and np.all(s >= math.log(50) - 1e-9)
    assert np.all(np.isfinite(spread)) and np.all(np.isfinite(spread_r)) and np.all(spread_r >= 0)


@pytest.mark.parametrize('lo,hi', [(-750.0, 750.0), (-1.0, 1.0), (-701.0, -699.0), (699.0, 701.0), (-6e-8, 6e-8)])
def test_members_exponential_over_the_range(lo, hi):
    """exp of a member's outputs (floor 0, albedo 1) against numpy's: an ulp of each."""
    import torch
    from monte_carlompi_gb300 import _abi
    n, bins = 40, surrogate.N_BRF
    ys = torch.linspace(lo, hi, n * bins).reshape(1, n, bins).half()
    if hi == 750:
        ys[0, 0, :3] = torch.tensor([float('nan'), float('inf'), float('-inf')])
    ys = torch.cat([ys, torch.zeros(1, n, 1).half()], 2).cuda().contiguous()
    mean, std = torch.zeros(1, 649, dtype=torch.float64, device='cuda'), torch.ones(1, 649, dtype=torch.float64, device='cuda')
    brf, alb = torch.empty((1, n, bins), dtype=torch.float64, device='cuda'), torch.empty((1, n), dtype=torch.float64, device='cuda')
    p = lambda t: t.data_ptr()  # noqa: E731
    assert _abi.load().mcw_brf_members(p(ys), 649, 1, n, p(mean), p(std), 0.0, p(brf), p(alb), surrogate._stream(torch)) == 0
    with np.errstate(over='ignore', under='ignore'):
        ref = np.exp(ys[:, :, :bins].cpu().double().numpy())
    assert np.allclose(brf.cpu().numpy(), ref, rtol=4.45e-16, atol=1e-323, equal_nan=True)
    assert (alb.cpu().numpy() == 1).all()


@pytest.mark.parametrize('n,members', [(1, 1), (127, 3), (129, 5), (1000, 2)])
def test_retrieval_steps_match_numpy(n, members):
    """Inputs encoded on the device, the grid's best point and the damped step against
    surrogate.encode and inverse._gn_step: steps cut at both ends, equal, infinite and NaN costs.
    float32 inputs: one rounding of a float64 value that may differ by an ulp."""
    import ctypes
    import torch
    from monte_carlompi_gb300 import _abi
    rng = np.random.default_rng(n)
    L, st, p = _abi.load(), surrogate._stream(torch), lambda t: t.data_ptr()
    raw = surrogate.sample_inputs(n, n + 1)
    known = torch.from_numpy(np.ascontiguousarray(raw[:, 1:])).cuda()
    hull = (ctypes.c_double * 8)(*surrogate.hull())
    grid = np.linspace(*inverse.LOG_R, 16)
    grid_d = torch.from_numpy(grid).cuda()
    x = torch.empty((16 * n, 4), device='cuda')
    assert L.mcw_brf_encode(p(grid_d), 16, p(known), n, hull, p(x), st) == 0
    ref = surrogate.encode(np.repeat(np.exp(grid), n), *np.tile(raw[:, 1:], (16, 1)).T)
    assert np.allclose(x.cpu().numpy(), ref, rtol=1.2e-7, atol=1e-7)
    cost = rng.random((16, n))
    cost[3, 0], cost[7:, n // 2], cost[:, n - 1] = np.nan, cost[7, n // 2], (np.inf if n > 1 else cost[:, 0])
    s = torch.empty(n, dtype=torch.float64, device='cuda')
    x1, x16 = torch.empty((n, 4), device='cuda'), torch.zeros((members, n, 8), dtype=torch.bfloat16, device='cuda')
    jtr, jtj = rng.normal(size=n) * 10, rng.random(n) * np.where(np.arange(n) % 3, 10.0, 0.1)
    cost_d, jtr_d, jtj_d = (torch.from_numpy(v).cuda() for v in (cost, jtr, jtj))

    def step(c):
        assert L.mcw_brf_gn_step(c, p(grid_d), 16, p(jtr_d), p(jtj_d), 1e-3, 0.7, *inverse.LOG_R, p(known), n, hull, p(s),
                                 p(x1), p(x16), members, st) == 0
        assert torch.equal(x16[:, :, :4], x1.to(torch.bfloat16).expand(members, n, 4)) and not x16[:, :, 4:].any()
        assert np.allclose(x1.cpu().numpy(), surrogate.encode(np.exp(s.cpu().numpy()), *raw[:, 1:].T), rtol=1.2e-7, atol=1e-7)
        return s.cpu().numpy()
    best, want = np.full(n, np.inf), np.zeros(n)
    for g, c in zip(grid, cost):
        better = c < best
        best[better], want[better] = c[better], g
    got = step(p(cost_d))
    assert np.array_equal(got, want)
    for _ in range(3):
        want = inverse._gn_step(jtr, jtj, got)
        got = step(None)
        assert np.allclose(got, want, rtol=0, atol=1e-15)


@pytest.mark.parametrize('n,members,weighted', [(1, 1, True), (33, 3, False), (130, 5, True)])
def test_brf_kernels_match_numpy(n, members, weighted):
    """Members' BRFs, their mean and spread, grid costs, Gauss-Newton sums and spreads of log r_eff
    from random outputs against the array arithmetic, NaN kept where it arises."""
    import torch
    from monte_carlompi_gb300 import _abi
    g = torch.Generator().manual_seed(n + members)
    L, st = _abi.load(), surrogate._stream(torch)
    pitch, bins = 656, surrogate.N_BRF
    ys = (torch.randn(members, n, pitch, generator=g)).half().cuda()
    y, yd = torch.randn(members, n, 652, generator=g).cuda(), torch.randn(members, n, 652, generator=g).cuda()
    ys[0, n - 1, 5] = float('nan')
    mean, std = (torch.randn(members, 649, generator=g) * 0.1).double(), (torch.rand(members, 649, generator=g) * 0.3).double()
    obs = torch.rand(n, bins, generator=g).double()
    share = surrogate.bin_weights()
    photons, rel = (1e6, 0.01) if weighted else (0.0, 0.0)
    new = lambda *shape: torch.empty(shape, dtype=torch.float64, device='cuda')  # noqa: E731
    p = lambda t: t.data_ptr()  # noqa: E731
    md, sd, od, wd = mean.cuda(), std.cuda(), obs.cuda(), torch.from_numpy(share).cuda()
    brf, alb, mu, am, sp = new(members, n, bins), new(members, n), new(n, bins), new(n), new(n)
    cost, f, j, v, sums = new(n), new(n, bins), new(n, bins), new(n, bins), new(2, n)
    spread, sigma = new(n), new(n)
    fl = surrogate.BRF_FLOOR
    assert L.mcw_brf_members(p(ys), pitch, members, n, p(md), p(sd), fl, p(brf), p(alb), st) == 0
    assert L.mcw_brf_stats(p(brf), p(alb), members, n, p(wd), p(mu), p(am), p(sp), st) == 0
    assert L.mcw_brf_cost(p(ys), pitch, members, 1, n, p(md), p(sd), fl, p(od), p(wd), photons, rel, p(cost), st) == 0
    assert L.mcw_brf_jacobian(p(y), p(yd), 652, members, n, p(md), p(sd), fl, p(f), p(j), p(v), p(od), p(wd), photons,
                              rel, p(sums[0]), p(sums[1]), st) == 0
    assert L.mcw_brf_logr(p(brf), p(mu), members, n, p(f), p(j), p(v), p(wd), photons, rel, p(spread), p(sigma), st) == 0
    torch.cuda.synchronize()
    o = ys[:, :, :649].cpu().double().numpy() * std.numpy()[:, None] + mean.numpy()[:, None]
    rb, ra = zip(*[surrogate.from_target(q) for q in o])
    rb, ra = np.stack(rb), np.stack(ra)
    ok = dict(rtol=1e-11, atol=1e-13, equal_nan=True)
    assert np.allclose(brf.cpu(), rb, **ok) and np.allclose(alb.cpu(), ra, **ok)
    m = rb.mean(0)
    assert np.allclose(mu.cpu(), m, **ok) and np.allclose(am.cpu(), ra.mean(0), **ok)
    assert np.allclose(sp.cpu(), np.sqrt((rb.std(0) ** 2 * share).sum(1) / (m ** 2 * share).sum(1)), **ok)
    on = obs.numpy()
    w0 = 1 / inverse.noise_variance(on, photons, rel) if weighted else share[None]
    assert np.allclose(cost.cpu(), (w0 * (m - on) ** 2).sum(1), **ok)
    yp = y[:, :, :649].cpu().double().numpy() * std.numpy()[:, None] + mean.numpy()[:, None]
    dp = yd[:, :, :649].cpu().double().numpy() * std.numpy()[:, None]
    a, shape = np.exp(yp[..., bins:]), np.exp(yp[..., :bins])
    fm = (shape - fl) * a
    jm = shape * dp[..., :bins] * a + (shape - fl) * (a * dp[..., bins:])
    rf, rj = fm.mean(0), jm.mean(0)
    rv = np.maximum((fm ** 2).mean(0) - rf ** 2, 0)
    assert np.allclose(f.cpu(), rf, **ok) and np.allclose(j.cpu(), rj, **ok)
    assert np.allclose(v.cpu(), rv, rtol=1e-6, atol=1e-13)
    vk = v.cpu().numpy()
    w = 1 / inverse.noise_variance(rf, photons, rel, vk) if weighted else np.broadcast_to(share[None], rf.shape)
    wn = 1 / inverse.noise_variance(rf, photons, rel) if weighted else share[None]
    assert np.allclose(sums[0].cpu(), (w * rj * (rf - on)).sum(1), rtol=1e-9, atol=1e-9 * np.abs(w * rj * rf).sum(1).max())
    assert np.allclose(sums[1].cpu(), (w * rj * rj).sum(1), rtol=1e-9)
    got = spread.cpu().numpy()
    assert np.allclose(got, inverse.logr_spread(rb, rj, w), rtol=1e-8, atol=1e-13, equal_nan=True)
    assert np.allclose(sigma.cpu(), 1 / np.sqrt((wn * rj * rj).sum(1)), rtol=1e-9)


def test_retrieval_refuses_arrays_of_other_shapes(trained):
    ens = trained[0]
    for obs, known in ((np.ones((4, 640)), np.ones((4, 3))), (np.ones((4, 648)), np.ones((3, 3))),
                       (np.ones((4, 648)), np.ones((4, 2)))):
        with pytest.raises(ValueError):
            inverse.surrogate_gn(ens, obs, known)


def test_retrieval_takes_noise_per_bin_and_per_observation(trained):
    """obs_noise as an array: the same number in every place is the number, in every form that
    broadcasts; a noise of each observation's own is that of a retrieval of it alone (its rows of the
    network and of the sums do not depend on the others); a noise per bin weights the costs, the
    Gauss-Newton sums and the spreads as the array arithmetic does."""
    from monte_carlompi_gb300 import _abi
    ens, ds, hold = trained
    n, rng = 7, np.random.default_rng(11)
    known, photons = ds.raw[:n, 1:], 1e6
    obs = ds.brf[:n] * (1 + 0.02 * rng.standard_normal((n, surrogate.N_BRF)))

    def solve(noise, rows=slice(None), **kw):
        return inverse.surrogate_gn(ens, obs[rows], known[rows], obs_photons=kw.get('photons', photons),
                                    obs_noise=noise, with_noise=True)
    want = solve(0.02)
    for shape in ((1,), (1, 1), (surrogate.N_BRF,), (1, surrogate.N_BRF), (n, 1), (n, surrogate.N_BRF)):
        for a, b in zip(solve(np.full(shape, 0.02)), want):
            assert np.array_equal(a, b), shape
    for a, b in zip(solve(0.02, photons=np.array([photons])), want):
        assert np.array_equal(a, b)
    for a, b in zip(solve(np.full((n, 1), 0.3), photons=None), solve(0.0, photons=None)):
        assert np.array_equal(a, b)
    each = np.linspace(0.005, 0.1, n)
    got = solve(each[:, None])
    for i in range(n):
        for a, b in zip(got, solve(float(each[i]), slice(i, i + 1))):
            assert np.allclose(a[i], b[0], rtol=1e-9, atol=1e-12), i
    with pytest.raises(ValueError):
        solve(np.ones((n + 1, 1)))
    # the kernels against the array arithmetic (test_brf_kernels_match_numpy's tolerances)
    rel = rng.uniform(0.0, 0.2, (n, surrogate.N_BRF))
    m, bins = 3, surrogate.N_BRF
    g = torch.Generator().manual_seed(5)
    ys = torch.randn(m, n, 656, generator=g).half().cuda()
    y, yd = torch.randn(m, n, 652, generator=g).cuda(), torch.randn(m, n, 652, generator=g).cuda()
    mean, std = torch.zeros(m, 649, dtype=torch.float64, device='cuda'), torch.full((m, 649), 0.2, dtype=torch.float64, device='cuda')
    od, wd, rd = (torch.from_numpy(np.ascontiguousarray(t)).cuda() for t in (obs, surrogate.bin_weights(), rel))
    new = lambda *shape: torch.empty(shape, dtype=torch.float64, device='cuda')  # noqa: E731
    p, fl, st = (lambda t: t.data_ptr()), surrogate.BRF_FLOOR, surrogate._stream(torch)  # noqa: E731
    brf, alb, mu, am, sp = new(m, n, bins), new(m, n), new(n, bins), new(n), new(n)
    cost, f, j, v, sums, spread, sigma = new(n), new(n, bins), new(n, bins), new(n, bins), new(2, n), new(n), new(n)
    L = _abi.load()
    assert L.mcw_brf_members(p(ys), 656, m, n, p(mean), p(std), fl, p(brf), p(alb), st) == 0
    assert L.mcw_brf_stats(p(brf), p(alb), m, n, p(wd), p(mu), p(am), p(sp), st) == 0
    assert L.mcw_brf_cost_noise(p(ys), 656, m, 1, n, p(mean), p(std), fl, p(od), p(wd), photons, p(rd), p(cost), st) == 0
    assert L.mcw_brf_jacobian_noise(p(y), p(yd), 652, m, n, p(mean), p(std), fl, p(f), p(j), p(v), p(od), p(wd), photons,
                                    p(rd), p(sums[0]), p(sums[1]), st) == 0
    assert L.mcw_brf_logr_noise(p(brf), p(mu), m, n, p(f), p(j), p(v), p(wd), photons, p(rd), p(spread), p(sigma), st) == 0
    rb, rmu, rf, rj, rv = (t.cpu().numpy() for t in (brf, mu, f, j, v))
    w0, w = 1 / inverse.noise_variance(obs, photons, rel), 1 / inverse.noise_variance(rf, photons, rel, rv)
    assert np.allclose(cost.cpu(), (w0 * (rmu - obs) ** 2).sum(1), rtol=1e-11, atol=1e-13)
    assert np.allclose(sums[0].cpu(), (w * rj * (rf - obs)).sum(1), rtol=1e-9, atol=1e-9 * np.abs(w * rj * rf).sum(1).max())
    assert np.allclose(sums[1].cpu(), (w * rj * rj).sum(1), rtol=1e-9)
    assert np.allclose(spread.cpu(), inverse.logr_spread(rb, rj, w), rtol=1e-8, atol=1e-13)
    wn = 1 / inverse.noise_variance(rf, photons, rel)
    assert np.allclose(sigma.cpu(), 1 / np.sqrt((wn * rj * rj).sum(1)), rtol=1e-9)


@pytest.mark.parametrize('members', [1024, 1025, 3037, 4096, 12800])
def test_costs_and_slopes_of_many_members(members):
    """The kernels that keep a share of every member in shared memory, past 48 KB of it, against the
    array arithmetic; a member more than they hold is refused."""
    from monte_carlompi_gb300 import _abi
    n, bins, fl, L, st = 2, surrogate.N_BRF, surrogate.BRF_FLOOR, _abi.load(), surrogate._stream(torch)
    g = torch.Generator().manual_seed(members)
    y, yd = torch.randn(members, n, 652, generator=g).half(), torch.randn(members, n, 652, generator=g)
    ys, y32, ydd = y.cuda(), y.float().cuda(), yd.cuda()
    mean, std = torch.zeros(members, 649, dtype=torch.float64, device='cuda'), torch.full((members, 649), 0.2, dtype=torch.float64, device='cuda')
    obs = torch.rand(n, bins, generator=g).double()
    od, wd = obs.cuda(), torch.from_numpy(surrogate.bin_weights()).cuda()
    new = lambda *shape: torch.empty(shape, dtype=torch.float64, device='cuda')  # noqa: E731
    p = lambda t: t.data_ptr()  # noqa: E731
    cost, f, j, v, sums = new(n), new(n, bins), new(n, bins), new(n, bins), new(2, n)

    def run(k):
        return (L.mcw_brf_cost(p(ys), 652, k, 1, n, p(mean), p(std), fl, p(od), p(wd), 0.0, 0.0, p(cost), st),
                L.mcw_brf_jacobian(p(y32), p(ydd), 652, k, n, p(mean), p(std), fl, p(f), p(j), p(v), p(od), p(wd), 0.0, 0.0,
                                   p(sums[0]), p(sums[1]), st))
    assert run(members) == (0, 0) and run(12801) == (-1, -1)
    torch.cuda.synchronize()
    yp, dp = y[:, :, :649].double().numpy() * 0.2, yd[:, :, :649].double().numpy() * 0.2
    a, shape = np.exp(yp[..., bins:]), np.exp(yp[..., :bins])
    rf = ((shape - fl) * a).mean(0)
    rj = (shape * dp[..., :bins] * a + (shape - fl) * (a * dp[..., bins:])).mean(0)
    # (sums of some thousand terms of the order of one, in another order than numpy's)
    assert np.allclose(f.cpu(), rf, rtol=1e-11, atol=1e-13) and np.allclose(j.cpu(), rj, rtol=1e-10, atol=1e-12)
    share = surrogate.bin_weights()
    assert np.allclose(cost.cpu(), (share * (rf - obs.numpy()) ** 2).sum(1), rtol=1e-10)
    assert np.allclose(sums[1].cpu(), (share * rj * rj).sum(1), rtol=1e-9)


@pytest.mark.parametrize('lo,hi', [(-700.0, 700.0), (-12.0, 4.0), (-0.01, 0.01)])
def test_members_exponential_to_half_an_ulp(lo, hi):
    """exp of the members' outputs (floor 0, albedo 1) against extended precision: half an ulp, and 0.05
    for the table's second part, the series (0.02), the reduced argument and three roundings of 2^-7 of
    the result."""
    from monte_carlompi_gb300 import _abi
    n, bins = 200, surrogate.N_BRF
    x = np.random.default_rng(8).uniform(lo, hi, (n, 649))
    x[:, bins] = 0.0
    ys = torch.zeros(n, 1, 656, dtype=torch.float16, device='cuda')            # n members, a row each
    mean, std = torch.from_numpy(x).cuda(), torch.ones(n, 649, dtype=torch.float64, device='cuda')
    brf, alb = torch.empty((n, bins), dtype=torch.float64, device='cuda'), torch.empty(n, dtype=torch.float64, device='cuda')
    p = lambda t: t.data_ptr()  # noqa: E731
    assert _abi.load().mcw_brf_members(p(ys), 656, n, 1, p(mean), p(std), 0.0, p(brf), p(alb), surrogate._stream(torch)) == 0
    got, want = brf.cpu().numpy().astype(np.longdouble), np.exp(x[:, :bins].astype(np.longdouble))
    ulp = np.ldexp(np.longdouble(1), np.frexp(want)[1] - 53)
    assert (np.abs(got - want) / ulp).max() <= 0.55
    assert (alb.cpu() == 1).all()


@pytest.mark.parametrize('members', [1, 2, 3, 5, 7, 1000])
def test_means_over_the_members_lose_nothing(members):
    """Means over the members are the sums divided, to the last bit, infinities kept; and a grid cost of
    BRFs next to 0 (exponentials next to the floor) keeps the digits of the members' own BRFs."""
    from monte_carlompi_gb300 import _abi
    n, bins, L, st = 6, surrogate.N_BRF, _abi.load(), surrogate._stream(torch)
    rng, p = np.random.default_rng(members), lambda t: t.data_ptr()
    new = lambda *shape: torch.empty(shape, dtype=torch.float64, device='cuda')  # noqa: E731
    y = torch.from_numpy(rng.uniform(-3, 3, (1, n, 652)).astype(np.float32))
    y[:, :, bins] = 0.0                                                        # albedo 1
    y[0, 0, 0] = 800.0
    yd = torch.ones(1, n, 652)
    yd[:, :, bins] = 0.0

    def slopes(k):
        ys, yds = y.expand(k, n, 652).contiguous().cuda(), yd.expand(k, n, 652).contiguous().cuda()
        mean, std, f, j, v = torch.zeros(k, 649, dtype=torch.float64, device='cuda'), \
            torch.ones(k, 649, dtype=torch.float64, device='cuda'), new(n, bins), new(n, bins), new(n, bins)
        assert L.mcw_brf_jacobian(p(ys), p(yds), 652, k, n, p(mean), p(std), 0.0, p(f), p(j), p(v), None, None, 0.0, 0.0,
                                  None, None, st) == 0
        return f.cpu().numpy(), j.cpu().numpy()
    f1, j1 = slopes(1)
    total = lambda t: np.add.accumulate(np.broadcast_to(t, (members, *t.shape)), 0)[-1]  # noqa: E731
    f, j = slopes(members)
    assert np.array_equal(f, total(f1) / members) and np.isinf(f[0, 0])
    assert np.array_equal(j, total(j1) / members, equal_nan=True) and np.isnan(j).sum() == 1   # (infinity times 0)
    # BRFs of 1e-11
    fl = surrogate.BRF_FLOOR
    mean = math.log(fl) + rng.uniform(-1e-9, 1e-9, (members, 649))
    mean[:, bins] = -0.3
    mean, std = torch.from_numpy(mean).cuda(), torch.ones(members, 649, dtype=torch.float64, device='cuda')
    ys = torch.zeros(members, 1, 656, dtype=torch.float16, device='cuda')
    brf, alb, cost = new(members, 1, bins), new(members, 1), new(1)
    obs, share = torch.zeros(1, bins, dtype=torch.float64, device='cuda'), torch.from_numpy(surrogate.bin_weights()).cuda()
    assert L.mcw_brf_members(p(ys), 656, members, 1, p(mean), p(std), fl, p(brf), p(alb), st) == 0
    assert L.mcw_brf_cost(p(ys), 656, members, 1, 1, p(mean), p(std), fl, p(obs), p(share), 0.0, 0.0, p(cost), st) == 0
    # (bins' means may cancel to a thousandth of their terms, each rounded once here and there)
    want = (surrogate.bin_weights() * brf.cpu().numpy()[:, 0].mean(0) ** 2).sum()
    assert abs(cost.item() / want - 1) < 1e-10


def test_albedos_to_half_an_ulp():
    """The members' albedos, as close to the exponential as the bins' (test_members_exponential_to_half_an_ulp)."""
    from monte_carlompi_gb300 import _abi
    n, bins = 20000, surrogate.N_BRF
    x = np.random.default_rng(9).uniform(-9.0, 0.0, n)
    mean = torch.zeros(n, 649, dtype=torch.float64, device='cuda')
    mean[:, bins] = torch.from_numpy(x).cuda()
    ys, std = torch.zeros(4000, 1, 656, dtype=torch.float16, device='cuda'), torch.ones(4000, 649, dtype=torch.float64, device='cuda')
    alb, brf = torch.empty(n, dtype=torch.float64, device='cuda'), torch.empty((4000, bins), dtype=torch.float64, device='cuda')
    p = lambda t: t.data_ptr()  # noqa: E731
    for lo in range(0, n, 4000):
        assert _abi.load().mcw_brf_members(p(ys), 656, 4000, 1, p(mean[lo:]), p(std), 0.0, p(brf), p(alb[lo:]),
                                           surrogate._stream(torch)) == 0
    got, want = alb.cpu().numpy().astype(np.longdouble), np.exp(x.astype(np.longdouble))
    ulp = np.ldexp(np.longdouble(1), np.frexp(want)[1] - 53)
    assert (np.abs(got - want) / ulp).max() <= 0.55
