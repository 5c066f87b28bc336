"""Grain-size retrieval: batched Gauss-Newton on log r_eff through the BRF surrogate.

Given observed 648-bin BRFs with known wavelength, incident zenith and depth,
find r_eff.  Each iteration evaluates the ensemble and the Jacobian
d BRF / d log r_eff in forward mode through the surrogate's tensor-core kernels
(`surrogate.forward_tangent`: the input is one scalar, so one tangent pass replaces a
backward pass per output bin).  Retrievals whose ensemble spread at the solution
exceeds ``spread_tol`` fall back to plain Monte Carlo: the same Gauss-Newton
iteration with BRFs and central-difference Jacobians from the GPU walk.  The spread
is either that of the members' BRFs (criterion 'brf': weighted RMS of their standard
deviation over the weighted RMS BRF) or that of the retrieved quantity (criterion
'r_eff': each member's BRF, taken through the Gauss-Newton normal equation at the
solution, gives the log r_eff that member would move the answer to; their standard
deviation is the surrogate's own relative uncertainty in r_eff).  The reference has no inverse; this consumes the same BRF definition
(post_processing.py:73-81, 2-D form).
"""
import ctypes
import math
import time

import numpy as np

from . import _abi
from . import surrogate as S

LOG_R = (math.log(S.R_RANGE[0]), math.log(S.R_RANGE[1]))
DAMPING, MAX_STEP = 1e-3, 0.7


def noise_variance(f, photons, rel_noise=0.0, model_var=None):
    """Per-bin variance of a BRF about the model value f [n, 648]: the counting noise of
    a walk of `photons` photons (the bin holds photons * w_b * BRF_b of them, w_b its
    expected share, so Var BRF_b = BRF_b / (photons * w_b)), relative Gaussian noise
    rel_noise, and the model's own per-bin variance when given."""
    wt = S.bin_weights()[None, :]
    v = np.maximum(f, 1e-3) / (photons * wt) + (rel_noise * f) ** 2
    return v + model_var if model_var is not None else v


def _ptr(t):
    return None if t is None else t.data_ptr()


class _Noise:
    """An observation's photons (0: none) and relative noise, one number or a torch CUDA float64
    [n, 648], as the kernels of csrc/brf.cu take them."""

    def __init__(self, photons, rel):
        self.photons, self.rel = photons, rel

    def entry(self, name):
        return getattr(_abi.load(), name if isinstance(self.rel, float) else name + '_noise')

    def args(self):
        return self.photons, self.rel if isinstance(self.rel, float) else _ptr(self.rel)


class _Slopes:
    """BRF, d BRF / d log r_eff and the members' variance of an ensemble at n points: one
    forward-mode pass of all members through the tensor-core kernels (the tangent of the first
    input, d x0 / d log r = 2 / (log r_max - log r_min)), then the chain rule through the target
    standardisation, exp and the albedo factor in one kernel."""

    def __init__(self, ens, n, scaling=None, share=None):
        import torch
        self.torch = torch
        self.n = n
        self.net = S.EnsembleTangent(torch, ens.members, n, 2.0 / (LOG_R[1] - LOG_R[0]))
        self.mean, self.std = ens.scaling() if scaling is None else scaling
        self.share = torch.from_numpy(S.bin_weights()).cuda() if share is None else share

    def at(self, s, known):
        """(f, j, v) torch CUDA float64 [n, 648] at log r = s (host arrays s [n], known [n, 3])."""
        return self.arrays(self.torch.from_numpy(S.encode(np.exp(s), *known.T)).cuda())

    def arrays(self, x=None):
        """(f, j, v) of inputs x, or of those the network's buffer holds."""
        f, j, v = (self.torch.empty((self.n, S.N_BRF), dtype=self.torch.float64, device=self.share.device) for _ in range(3))
        self._evaluate(x, f, j, v, None, _Noise(0.0, 0.0), None)
        return f, j, v

    def sums(self, obs, noise, out):
        """The sums over the bins of w j (f - obs) and w j^2 into out [2, n] (obs torch CUDA float64
        [n, 648]), of the inputs the network's buffer holds."""
        self._evaluate(None, None, None, None, obs, noise, out)

    def _evaluate(self, x, f, j, v, obs, noise, out):
        y, ydot = self.net.run(x)
        jtr, jtj = (None, None) if out is None else (out[0], out[1])
        rc = noise.entry('mcw_brf_jacobian')(_ptr(y), _ptr(ydot), y.shape[2], y.shape[0], self.n, _ptr(self.mean),
                                             _ptr(self.std), S.BRF_FLOOR, _ptr(f), _ptr(j), _ptr(v), _ptr(obs),
                                             _ptr(self.share), *noise.args(), _ptr(jtr), _ptr(jtj),
                                             S._stream(self.torch))
        if rc:
            raise _abi.McwError(rc, 'mcw_brf_jacobian failed')


def _brf_and_jacobian(ens, s, known, chunk=16384, with_var=False):
    """Ensemble-mean BRF [n, 648] and d BRF / d log r [n, 648] at log r = s (_Slopes).  with_var:
    also the variance of the members' BRFs per bin."""
    n = s.shape[0]
    out = [np.zeros((n, S.N_BRF)) for _ in range(3)]
    slopes = None
    for lo in range(0, n, chunk):
        hi = min(n, lo + chunk)
        if slopes is None or slopes.n != hi - lo:
            slopes = _Slopes(ens, hi - lo)
        arrays = slopes.at(s[lo:hi], known[lo:hi])
        for o, t in zip(out, arrays):
            o[lo:hi] = t.cpu().numpy()
    return tuple(out) if with_var else tuple(out[:2])


def _gn_update(f, jac, obs, s, w, damping=DAMPING, max_step=MAX_STEP):
    r = f - obs
    return _gn_step((w * jac * r).sum(1), (w * jac * jac).sum(1), s, damping, max_step)


def _gn_step(jtr, jtj, s, damping=DAMPING, max_step=MAX_STEP):
    step = -jtr / (jtj * (1 + damping) + 1e-30)
    step = np.clip(step, -max_step, max_step)
    return np.clip(s + step, LOG_R[0], LOG_R[1])


def logr_spread(f_members, jac, w):
    """Standard deviation over the members of the log r_eff shift that takes the
    ensemble-mean BRF to each member's BRF, linearised at the solution:
    ds_m = sum_b w_b J_b (f_mb - mean_b) / sum_b w_b J_b^2.  f_members [M, n, bins],
    jac [n, bins] (d BRF / d log r), w [1, bins] or [bins]."""
    dev = f_members - f_members.mean(0, keepdims=True)
    ds = (w * jac * dev).sum(2) / np.maximum((w * jac * jac).sum(1), 1e-300)
    return ds.std(0)


def surrogate_gn(ens, obs, known, iters=6, obs_photons=None, obs_noise=0.0, with_noise=False):
    """Gauss-Newton on s = log r_eff through the surrogate; starts from the best of a
    16-point grid.  With obs_photons, every bin's residual is weighted by the inverse of
    its variance (noise_variance: the observation's counting noise for obs_photons
    photons and its relative noise obs_noise, a number or an array that broadcasts to
    obs's shape, plus the ensemble's variance in that bin);
    without, by the bin's photon share.  Returns (s, brf at s, BRF spread at s, log r_eff
    spread at s) and, with with_noise, the posterior width of s from the observation
    noise alone, 1 / sqrt(sum_b J_b^2 / var_b)."""
    if obs.ndim != 2 or obs.shape[1] != S.N_BRF or np.shape(known) != (obs.shape[0], 3):
        raise ValueError('obs must be [n, %d] and known [n, 3]' % S.N_BRF)
    photons = np.asarray(obs_photons or 0, np.float64).item()
    rel = np.asarray(obs_noise if photons else 0, np.float64)        # (weights without photons take no noise)
    rel = rel.item() if rel.size == 1 else np.broadcast_to(rel, obs.shape)
    parts = [_surrogate_gn(ens, obs[lo:lo + 4096], known[lo:lo + 4096], iters, photons,
                           rel if isinstance(rel, float) else rel[lo:lo + 4096])
             for lo in range(0, obs.shape[0], 4096)]
    if not parts:
        parts = [(np.zeros(0), np.zeros((0, S.N_BRF)), np.zeros(0), np.zeros(0), np.zeros(0))]
    out = tuple(np.concatenate([p[k] for p in parts]) for k in range(5))
    return out if with_noise else out[:4]


def _surrogate_gn(ens, obs, known, iters, photons, rel):
    """surrogate_gn of a few thousand observations, queued on the device from the grid to the
    spreads (FP64, csrc/brf.cu) without the host waiting in between."""
    import torch
    n = obs.shape[0]
    f64 = dict(dtype=torch.float64, device='cuda')
    known_d = torch.from_numpy(np.ascontiguousarray(known, np.float64)).cuda()
    obs_d = torch.from_numpy(np.ascontiguousarray(obs, np.float64)).cuda()
    share = torch.from_numpy(S.bin_weights()).cuda()
    noise = _Noise(photons, rel if isinstance(rel, float) else torch.from_numpy(np.array(rel)).cuda())
    mean, std = ens.scaling()
    L, st, k = _abi.load(), S._stream(torch), len(ens.members)
    hull = (ctypes.c_double * 8)(*S.hull())

    def check(rc, what):
        if rc:
            raise _abi.McwError(rc, '%s failed' % what)
    # the grid: every observation at every point in one forward pass
    grid = torch.from_numpy(np.linspace(LOG_R[0], LOG_R[1], 16)).cuda()
    x = torch.empty((16 * n, S.DIMS[0]), dtype=torch.float32, device='cuda')
    check(L.mcw_brf_encode(_ptr(grid), 16, _ptr(known_d), n, hull, _ptr(x), st), 'mcw_brf_encode')
    ys = ens.predict_std(x)
    cost = torch.empty((16, n), **f64)
    check(noise.entry('mcw_brf_cost')(_ptr(ys), ys.stride(1), k, 16, n, _ptr(mean), _ptr(std), S.BRF_FLOOR,
                                      _ptr(obs_d), _ptr(share), *noise.args(), _ptr(cost), st), 'mcw_brf_cost')
    # (laid out while the grid's costs are being worked out)
    slopes = _Slopes(ens, n, (mean, std), share)
    s, sums = torch.empty(n, **f64), torch.empty((2, n), **f64)
    x = torch.empty((n, S.DIMS[0]), dtype=torch.float32, device='cuda')

    def step(cost_p):
        check(L.mcw_brf_gn_step(cost_p, _ptr(grid), 16, _ptr(sums[0]), _ptr(sums[1]), DAMPING, MAX_STEP, LOG_R[0],
                                LOG_R[1], _ptr(known_d), n, hull, _ptr(s), _ptr(x), _ptr(slopes.net.x), k, st),
              'mcw_brf_gn_step')
    step(_ptr(cost))
    for _ in range(iters):
        slopes.sums(obs_d, noise, sums)
        step(None)
    brf, alb = ens._member_brfs(x, mean, std)
    pred, _, spread = ens._brf_stats(brf, alb, share)
    f, j, v = slopes.arrays()
    spread_r, sigma = torch.empty_like(spread), torch.empty_like(spread)
    check(noise.entry('mcw_brf_logr')(_ptr(brf), _ptr(pred), k, n, _ptr(f), _ptr(j), _ptr(v), _ptr(share),
                                      *noise.args(), _ptr(spread_r), _ptr(sigma), st), 'mcw_brf_logr')
    return tuple(t.cpu().numpy() for t in (s, pred, spread, spread_r, sigma))


def mc_gn(walker, obs, known, s0, n_photon=1000000, iters=3, h=0.05, seed=0x5EED0055, obs_photons=None,
          obs_noise=0.0):
    """Gauss-Newton on log r_eff with BRFs and central-difference Jacobians from the walk.
    With obs_photons the residuals are weighted by the inverse variance of the
    observation (noise_variance) plus the walk's own counting noise at n_photon."""
    share = S.bin_weights()[None, :]
    s = np.array(s0, dtype=np.float64)
    evals = 0
    for it in range(iters):
        rows = np.concatenate([np.column_stack([np.exp(s + d), known]) for d in (0.0, h, -h)])
        brf, _ = S.mc_brf(walker, rows, n_photon, seed + 1000 * it)
        evals += rows.shape[0]
        n = s.shape[0]
        f, fp, fm = brf[:n], brf[n:2 * n], brf[2 * n:]
        if obs_photons:
            w = 1.0 / (noise_variance(f, obs_photons, obs_noise) + noise_variance(f, n_photon))
        else:
            w = share
        s = _gn_update(f, (fp - fm) / (2 * h), obs, s, w)
    return s, evals


def mc_correct(ens, walker, obs, known, s0, iters=2, n_photon=1000000, seed=0x5EED0066, obs_photons=None,
               obs_noise=0.0):
    """Gauss-Newton on log r_eff whose residuals come from the walk and whose Jacobian
    comes from the surrogate: s <- s - sum w J (f_MC(s) - obs) / sum w J^2, J = d BRF /
    d log r of the ensemble at s.  One walk per retrieval and iteration (plain Monte
    Carlo Gauss-Newton needs three, for its central differences, and a grid search
    before); the answer converges to the Monte Carlo solution as fast as the network's
    Jacobian is close to the walk's (error times |1 - J_MC / J| per iteration), and the
    network's systematic BRF error drops out of the residual.  Returns (s, walks)."""
    share = S.bin_weights()[None, :]
    s = np.array(s0, dtype=np.float64)
    n = s.shape[0]
    evals = 0
    for it in range(iters):
        f, _ = S.mc_brf(walker, np.column_stack([np.exp(s), known]), n_photon, seed + 1000 * it)
        evals += n
        _, jac = _brf_and_jacobian(ens, s, known)
        if obs_photons:
            w = 1.0 / (noise_variance(f, obs_photons, obs_noise) + noise_variance(f, n_photon))
        else:
            w = share
        s = _gn_update(f, jac, obs, s, w)
    return s, evals


def mc_retrieve(walker, obs, known, grid=16, iters=4, n_photon=1000000, seed=0x5EED0077, obs_photons=None,
                obs_noise=0.0):
    """The same retrieval with plain Monte Carlo only: the 16-point log r_eff grid and the
    Gauss-Newton iterations evaluated by the walk, weighted as mc_gn.  Returns (s, BRF
    evaluations)."""
    n = obs.shape[0]
    w = 1.0 / noise_variance(obs, obs_photons, obs_noise) if obs_photons else S.bin_weights()[None, :]
    g = np.linspace(LOG_R[0], LOG_R[1], grid)
    rows = np.concatenate([np.column_stack([np.full(n, math.exp(v)), known]) for v in g])
    brf, _ = S.mc_brf(walker, rows, n_photon, seed)
    cost = np.stack([(w * (brf[k * n:(k + 1) * n] - obs) ** 2).sum(1) for k in range(grid)])
    s0 = g[np.argmin(cost, axis=0)]
    s, evals = mc_gn(walker, obs, known, s0, n_photon=n_photon, iters=iters, seed=seed + 1,
                     obs_photons=obs_photons, obs_noise=obs_noise)
    return s, evals + rows.shape[0]


def retrieve(ens, walker, obs, known, spread_tol=0.02, mc_photons=1000000, criterion='brf', obs_photons=None,
             obs_noise=0.0, kappa=1.0, fallback='gn', correct_iters=2):
    """Surrogate retrieval with Monte Carlo fallback.  Criterion 'brf': the ensemble
    spread of the BRF exceeds spread_tol; 'r_eff': the ensemble spread of the retrieved
    log r_eff exceeds spread_tol; 'posterior': the ensemble spread of log r_eff exceeds
    kappa times the posterior width the observation noise alone allows (the network's
    own uncertainty would dominate the error; needs obs_photons).  The fallback of a
    flagged retrieval: 'correct' (mc_correct: correct_iters walks at the surrogate's
    answer, the surrogate's Jacobian) or 'gn' (mc_gn: Monte Carlo Gauss-Newton with
    central differences).  With obs_photons the residuals of both paths are weighted by
    their inverse noise variance.  Returns dict of results and timings."""
    if criterion not in ('brf', 'r_eff', 'posterior'):
        raise ValueError("criterion must be 'brf', 'r_eff' or 'posterior'")
    if criterion == 'posterior' and not obs_photons:
        raise ValueError("the 'posterior' criterion needs obs_photons")
    if fallback not in ('gn', 'correct'):
        raise ValueError("fallback must be 'gn' or 'correct'")
    t0 = time.perf_counter()
    s, _, spread, spread_r, sigma = surrogate_gn(ens, obs, known, obs_photons=obs_photons, obs_noise=obs_noise,
                                                 with_noise=True)
    t_net = time.perf_counter() - t0
    if criterion == 'brf':
        flagged = spread > spread_tol
    elif criterion == 'r_eff':
        flagged = spread_r > spread_tol
    else:
        flagged = spread_r > kappa * sigma
    t0 = time.perf_counter()
    mc_evals = 0
    if np.any(flagged):
        if fallback == 'correct':
            s_mc, mc_evals = mc_correct(ens, walker, obs[flagged], known[flagged], s[flagged], iters=correct_iters,
                                        n_photon=mc_photons, obs_photons=obs_photons, obs_noise=obs_noise)
        else:
            s_mc, mc_evals = mc_gn(walker, obs[flagged], known[flagged], s[flagged], n_photon=mc_photons,
                                   obs_photons=obs_photons, obs_noise=obs_noise)
        s = s.copy()
        s[flagged] = s_mc
    t_mc = time.perf_counter() - t0
    return dict(r_eff=np.exp(s), flagged=flagged, spread=spread, spread_r_eff=spread_r, sigma_noise=sigma,
                seconds_net=t_net, seconds_mc=t_mc, mc_brf_evals=mc_evals, criterion=criterion, fallback=fallback)
