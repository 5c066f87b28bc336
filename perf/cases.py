"""What this framework is used for, as cases that can be timed and compared.

A case names a kind of work, its sizes and its options; `prepare` makes what a program holds
before the call (tables and configs on a Walker, a network, a training engine, records), `run`
makes one pass through the public entry points, `exact` gives the result in 64 bits where plain
torch or numpy can, `work` the bytes and operations that the pass cannot do without.

Kinds:
  walk      one config's photons through Walker.walk (FP32): what every run of the driver does
  sweep     many configs as one captured launch (Walker.graph): parameter sweeps
  pol       the polarised walk of aspherical grains (FP32)
  replay    the FP64 walk in the reference's arithmetic, plain or polarised: parity runs
  post      BRF and albedo from per-photon records
  forward   the surrogate network's predictions, one network or the whole ensemble
  train     Adam steps of an ensemble (one short epoch)
  grad      one network through torch autograd: outputs and every gradient
  retrieve  Gauss-Newton grain-size retrieval through the surrogate
"""
import math

import numpy as np
import torch

from monte_carlompi_gb300 import _abi, inverse, post, ssp
from monte_carlompi_gb300 import surrogate as S
from monte_carlompi_gb300.config import WalkConfig
from monte_carlompi_gb300.walker import Walker

WIDTHS = (4, 256, 256, 256, 649)
FLOP_ROW = 2 * sum(a * b for a, b in zip(WIDTHS[:-1], WIDTHS[1:]))     # one row forward
N_PARAMS = sum(a * b + b for a, b in zip(WIDTHS[:-1], WIDTHS[1:]))
OPS_PER_EVENT = 100             # thread instructions of one FP32 scatter event

# ---------------------------------------------------------------- the cases


def listed():
    return [
        # the smallest call: a trial run of a thousand photons, records wanted on the host;
        # launches, copies and host work are most of it
        dict(name='walk_1k', kind='walk', n=1000, r_um=100.0, wvl=1.30, theta0=0.0, depth=0.5, R=1.0,
             soot=0.0, records='host'),
        # an ordinary run: a thin, sooty layer over ground, photons counted in the hundred
        # thousands, records in the caller's own array
        dict(name='walk_soot_100k', kind='walk', n=100003, r_um=400.0, wvl=1.03, theta0=45.0, depth=0.02,
             R=0.25, soot=2e-7, records='host'),
        # the largest single run: a million photons of deep snow, records left on the device
        dict(name='walk_1m', kind='walk', n=1000000, r_um=250.0, wvl=1.55, theta0=60.0, depth=0.10, R=0.5,
             soot=0.0, records='device'),
        # a parameter sweep: 64 configs of very different photon counts and walk lengths
        dict(name='sweep_64', kind='sweep', n_cfg=64, lo=1e4, hi=1e6, pick=3, records='device'),
        # polarised walk of hexagonal plates over a partly reflecting ground
        dict(name='pol_200k', kind='pol', n=200000, re_um=120.0, wvl=1.30, theta0=30.0, tau=20.0, R=0.5),
        # the driver's default run in the reference's own arithmetic
        dict(name='replay_10k', kind='replay', n=10000, polarised=False, r_um=100.0, wvl=1.30, theta0=0.0,
             depth=0.5),
        # the post-processing of a million-photon run: the photodiode dome's zenith bins
        dict(name='post_1m', kind='post', n=1000000, n_bins=137, n_cfg=1, f64=False),
        # one network on a few hundred inputs in FP32: an interactive prediction
        dict(name='forward_300', kind='forward', rows=300, members=1, half=False),
        # the ensemble over a whole map of inputs, FP16 outputs
        dict(name='ensemble_64k', kind='forward', rows=65536, members=5, half=True),
        # training as the surrogate is trained: five members, batch 256
        dict(name='train_256', kind='train', members=5, batch=256, steps=4),
        # one network differentiated by autograd over a large batch
        dict(name='grad_64k', kind='grad', rows=65536, need_dx=False),
        # grain-size retrieval of a scene's observations through the surrogate
        dict(name='retrieve_128', kind='retrieve', n=128, members=5, weighted=True),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case: sizes over the ranges the listed ones stand for (log-uniform, odd ones
    among them), the options as they are met."""
    kind = rng.choice(['walk', 'walk', 'walk', 'sweep', 'pol', 'replay', 'post', 'forward', 'forward', 'train',
                       'grad', 'retrieve'])
    if kind == 'walk':
        return dict(kind=kind, n=int(_log(rng, 1, 1e6)), r_um=round(_log(rng, 50, 1500), 1),
                    wvl=round(rng.uniform(0.9, 1.8), 3), theta0=round(rng.uniform(0, 75), 1),
                    depth=round(_log(rng, 0.01, 1.0), 4), R=round(rng.uniform(0, 1), 2),
                    soot=rng.choice([0.0, 0.0, 1e-8, 5e-7]), records=rng.choice(['host', 'device', 'none']))
    if kind == 'sweep':
        return dict(kind=kind, n_cfg=rng.randint(2, 48), lo=1e3, hi=float(int(_log(rng, 1e4, 1e6))),
                    pick=rng.randrange(1, 1 << 20), records=rng.choice(['device', 'none']))
    if kind == 'pol':
        return dict(kind=kind, n=int(_log(rng, 100, 2e5)), re_um=rng.choice([60.0, 120.0, 250.0]),
                    wvl=rng.choice([1.1, 1.2, 1.3, 1.5, 1.7]), theta0=round(rng.uniform(0, 75), 1),
                    tau=round(_log(rng, 1, 60), 2), R=round(rng.uniform(0, 1), 2))
    if kind == 'replay':
        return dict(kind=kind, n=int(_log(rng, 50, 1e4)), polarised=rng.random() < 0.4,
                    r_um=round(_log(rng, 50, 1500), 1), wvl=rng.choice([1.2, 1.3, 1.5, 1.7]),
                    theta0=round(rng.uniform(0, 75), 1), depth=round(_log(rng, 0.01, 0.5), 4))
    if kind == 'post':
        return dict(kind=kind, n=int(_log(rng, 1e3, 1e6)), n_bins=rng.randint(18, 180),
                    n_cfg=rng.choice([1, 1, 3, 64]), f64=rng.random() < 0.3)
    if kind == 'forward':
        members = rng.choice([1, 1, 3, 5])
        return dict(kind=kind, rows=int(_log(rng, 1, 65536)), members=members,
                    half=members > 1 or rng.random() < 0.5)
    if kind == 'train':
        return dict(kind=kind, members=rng.randint(1, 5), batch=8 * int(_log(rng, 8, 512)),
                    steps=rng.randint(1, 4))
    if kind == 'grad':
        return dict(kind=kind, rows=int(_log(rng, 30, 65536)), need_dx=rng.random() < 0.4)
    return dict(kind=kind, n=int(_log(rng, 8, 128)), members=rng.choice([3, 5]), weighted=rng.random() < 0.7)


# ---------------------------------------------------------------- walks

RADII = (50.0, 100.0, 200.0, 400.0, 800.0, 1500.0)
FWHM = 0.085
PLATE_WVLS = [round(1.0 + 0.025 * i, 4) for i in range(41)]                                # um
PLATE_RE = (60.0, 120.0, 250.0)                                                            # um
PLATE_THETA = [0.5 * k for k in range(20)] + [10.0 + 2.0 * k for k in range(86)]           # deg
STOKES = (1.0, 0.3, 0.2, 0.1)


def _tau(depth, r_um):
    return depth * ssp.ext_cff_mss_sphere(r_um) * 300.0


def _sphere(c, n, **more):
    """A sphere config and its tables (synthetic formulas on the grid the driver reads)."""
    lo, hi = ssp.grid_for(c['wvl'], FWHM)
    cfg = WalkConfig(n_photon=n, wvl0=c['wvl'], half_width=FWHM, theta0_deg=c['theta0'],
                     tau_tot=_tau(c['depth'], c['r_um']), rds_snw=c['r_um'], **more)
    return cfg, ssp.synthetic_ice_table(c['r_um'], lo, hi), ssp.synthetic_impurity_table(lo, hi)


def _plates(c, n, tau, R):
    """A config of hexagonal plates with its SSP rows and phase matrices."""
    rows = ssp.synthetic_isca_rows(PLATE_WVLS, [c['re_um']])
    a = np.array(rows)
    ext = 1e6 * a[:, 3] * a[:, 4] / (917.0 * a[:, 2])
    ice = ssp.SSPTable(a[:, 0], a[:, 5], ext, a[:, 6], wvl_unit=ssp.WVL_MICRONS)
    els = ssp.synthetic_phase_rows(rows, PLATE_THETA)
    phase = ssp.phase_table([PLATE_THETA] * 6, [els[0]] + [e * els[0] for e in els[1:]], a[:, 0], c['wvl'])
    lo, hi = ssp.grid_for(c['wvl'], FWHM)
    cfg = WalkConfig(n_photon=n, wvl0=c['wvl'], half_width=FWHM, theta0_deg=c['theta0'], tau_tot=tau,
                     lambertian_reflectance=R, ssp_nearest=True, polarised=True, stokes0=STOKES)
    return cfg, ice, ssp.synthetic_impurity_table(lo, hi), phase


def _sweep_configs(c):
    rng = np.random.default_rng(c['pick'])
    cfgs = []
    for _ in range(c['n_cfg']):
        k = int(rng.integers(len(RADII)))
        cfgs.append(WalkConfig(n_photon=int(math.exp(rng.uniform(math.log(c['lo']), math.log(c['hi'])))),
                               wvl0=float(np.round(rng.uniform(0.9, 1.8), 3)), half_width=FWHM,
                               theta0_deg=float(rng.choice([0.0, 30.0, 45.0, 60.0])),
                               tau_tot=_tau(float(rng.choice([0.02, 0.10, 1.0])), RADII[k]),
                               lambertian_reflectance=0.5, ice_table=k, rds_snw=RADII[k]))
    return cfgs


def _events(n, coalbedo, tau):
    """About how many scatter events n photons have: absorption ends a walk in deep snow, the
    layer's faces one in a thin layer."""
    return n * min(4.4 / math.sqrt(max(coalbedo, 1e-7)), 1.0 + tau)


def _tallies(t):
    """A walk's tallies as plain integer arrays."""
    return {k: t[k].view(np.int64 if t[k].dtype.itemsize == 8 else np.int32)
            for k in ('n_cond', 'q_cond_fx', 'n_events', 'max_n_scat', 'bin_count', 'bin_wvn_fx')}


def _host_records(rec, more=()):
    return {k: rec[k] for k in ('condition', 'n_scat', 'wvn', 'theta_n', 'phi_n', 'path_length', 'snow_depth') + more}


def _device_records(buf):
    """RECORD32 rows in device memory: two integers, five floats, the config's index."""
    return {'counts': buf[:, :2], 'values': buf.view(torch.float32)[:, 2:7], 'config': buf[:, 7]}


# ---------------------------------------------------------------- the network


def _weights(seed, member):
    """FP32 weights and biases of one network, at the scale its initialisation gives."""
    g = torch.Generator(device='cuda').manual_seed(7919 * (seed % (1 << 40)) + member)
    out = []
    for k, n in zip(WIDTHS[:-1], WIDTHS[1:]):
        bound = math.sqrt(6.0 / k) if n != WIDTHS[-1] else math.sqrt(3.0 / k)
        out.append((torch.rand((n, k), generator=g, device='cuda') * 2 - 1) * bound)
        out.append((torch.rand(n, generator=g, device='cuda') * 2 - 1) * 0.1)
    return out


def _net(seed, member):
    net = S.SurrogateMLP(seed=member)
    for k, w in enumerate(_weights(seed, member)):
        net.params[k].copy_(w)
        if k % 2 == 0:
            net.w16[k // 2].copy_(w)
    return net


def _inputs(seed, rows):
    g = torch.Generator(device='cuda').manual_seed(104729 * (seed % (1 << 40)) + 1)
    return torch.rand((rows, WIDTHS[0]), generator=g, device='cuda') * 2 - 1


def _targets(seed, rows):
    g = torch.Generator(device='cuda').manual_seed(15485863 * (seed % (1 << 36)) + 2)
    return torch.randn((rows, WIDTHS[-1]), generator=g, device='cuda')


def _loss_weights():
    """Loss weights of the outputs: bins by their photon share (mean 1), the albedo 10."""
    mids = (np.arange(18) + 0.5) * (np.pi / 36)
    w = np.repeat(np.sin(mids) * np.cos(mids), 36)
    return np.concatenate([w / w.mean(), [10.0]]).astype(np.float32)


def _mlp64(x, params):
    h = x
    for k in range(0, 8, 2):
        h = h @ params[k].T + params[k + 1]
        if k < 6:
            h = h * torch.sigmoid(h)
    return h


# ---------------------------------------------------------------- prepare


def _prepare_walk(c, seed):
    cfg, ice, imp = _sphere(c, c['n'], lambertian_reflectance=c['R'], imp_cnc=c['soot'])
    w = Walker(0)
    w.set_tables([ice], imp)
    s = dict(w=w, cfgs=[cfg], seed=seed, records=c['records'])
    if c['records'] == 'host':
        s['out'] = np.zeros(c['n'], _abi.RECORD32)
    elif c['records'] == 'device':
        s['buf'] = torch.zeros((c['n'], 8), dtype=torch.int32, device='cuda')
    return s


def _prepare_sweep(c, seed):
    cfgs = _sweep_configs(c)
    w = Walker(0)
    w.set_tables([ssp.synthetic_ice_table(r, 600, 2100) for r in RADII], ssp.synthetic_impurity_table(600, 2100))
    s = dict(w=w, seed=seed)
    if c['records'] == 'device':
        s['buf'] = torch.zeros((sum(x.n_photon for x in cfgs), 8), dtype=torch.int32, device='cuda')
    s['graph'] = w.graph(cfgs, device_ptr=s['buf'].data_ptr() if 'buf' in s else None)
    return s


def _prepare_pol(c, seed):
    cfg, ice, imp, phase = _plates(c, c['n'], c['tau'], c['R'])
    w = Walker(0)
    w.set_tables([ice], imp)
    w.set_phase_matrices([phase])
    return dict(w=w, cfgs=[cfg], seed=seed, out=np.zeros(c['n'], _abi.RECORD32P))


def _prepare_replay(c, seed):
    w = Walker(0)
    if c['polarised']:
        cfg, ice, imp, phase = _plates(dict(c, re_um=min(PLATE_RE, key=lambda r: abs(r - c['r_um']))), c['n'],
                                       min(40.0, _tau(c['depth'], c['r_um'])), 0.5)
        w.set_tables([ice], imp)
        w.set_phase_matrices([phase])
    else:
        cfg, ice, imp = _sphere(c, c['n'])
        w.set_tables([ice], imp)
    return dict(w=w, cfgs=[cfg], seed=seed, mode='pol64' if c['polarised'] else 'replay64')


def _records(c, seed):
    """Records as a walk leaves them: most photons leave at the top or are absorbed, exits
    spread over the hemisphere by their solid angle, wavenumbers on the 0.01 um grid."""
    rng = np.random.default_rng(seed)
    n = c['n']
    rec = np.zeros(n, _abi.RECORD64 if c['f64'] else _abi.RECORD32)
    rec['condition'] = rng.choice([1, 2, 3, 4, 5], n, p=[0.48, 0.07, 0.01, 0.42, 0.02])
    rec['n_scat'] = rng.geometric(1 / 37.0, n)
    rec['wvn'] = 1.0 / (np.rint(100 * rng.normal(1.3, 0.036, n)) / 100)
    rec['theta_n'] = 0.5 * np.arccos(1 - 2 * rng.random(n))
    rec['phi_n'] = rng.random(n) * 2 * np.pi
    rec['path_length'] = rng.exponential(0.02, n)
    rec['snow_depth'] = 0.1
    if c['n_cfg'] > 1:
        rec['config'] = np.sort(rng.integers(0, c['n_cfg'], n))
    return rec


def _prepare_forward(c, seed):
    nets = [_net(seed, k) for k in range(c['members'])]
    s = dict(x=_inputs(seed, c['rows']), half=c['half'])
    if c['members'] == 1:
        s['net'] = nets[0]
        nets[0].packed()
    else:
        s['ens'] = S.Ensemble(nets)
        s['ens'].packed()
    return s


def _perms(c, seed):
    rng = np.random.default_rng(seed)
    return [rng.permutation(c['batch'] * c['steps']) for _ in range(c['members'])]


def _prepare_train(c, seed):
    rows = c['batch'] * c['steps']
    tr = S.EnsembleTrainer([_net(seed, k) for k in range(c['members'])], c['batch'], _inputs(seed, rows),
                           _targets(seed, rows), torch.from_numpy(_loss_weights()).cuda(), lr=1e-3)
    return dict(tr=tr, perms=_perms(c, seed), steps=c['steps'])


def _prepare_grad(c, seed):
    return dict(x=_inputs(seed, c['rows']).requires_grad_(c['need_dx']),
                params=[w.requires_grad_(True) for w in _weights(seed, 0)], gy=_targets(seed, c['rows']) / c['rows'])


def _prepare_retrieve(c, seed):
    nets = [_net(seed, k) for k in range(c['members'])]
    rng = np.random.default_rng(seed)
    raw = np.column_stack([np.exp(rng.uniform(math.log(50.0), math.log(1500.0), c['n'])),
                           rng.uniform(0.9, 1.8, c['n']), rng.uniform(0.3, 1.0, c['n']),
                           np.exp(rng.uniform(math.log(0.01), 0.0, c['n']))])
    # targets' scaling as training leaves it: log(BRF / albedo + floor) about 0, log(albedo) below
    mean = torch.zeros(649, dtype=torch.float64, device='cuda')
    mean[648] = -0.7
    std = torch.full((649,), 0.25, dtype=torch.float64, device='cuda')
    for m in nets:
        m.y_mean, m.y_std = mean.clone(), std.clone()
    # observations: the members' mean at the hidden grain sizes, with 1% noise
    x = np.stack([2 * np.log(raw[:, 0] / 50.0) / math.log(30.0) - 1, 2 * (raw[:, 1] - 0.9) / 0.9 - 1,
                  2 * (raw[:, 2] - 0.3) / 0.7 - 1, 2 * np.log(raw[:, 3] / 0.01) / math.log(100.0) - 1], axis=1)
    x = torch.from_numpy(x).cuda()
    brf = 0
    for m in nets:
        y = _mlp64(x, [p.double() for p in m.params]) * std + mean
        brf = brf + (torch.exp(y[:, :648]) - 0.02) * torch.exp(y[:, 648:]) / len(nets)
    obs = np.maximum(brf.cpu().numpy(), 0) * (1 + 0.01 * rng.standard_normal((c['n'], 648)))
    return dict(ens=S.Ensemble(nets), obs=obs, known=raw[:, 1:],
                noise=dict(obs_photons=1000000, obs_noise=0.01) if c['weighted'] else {})


def prepare(case, seed):
    kind = case['kind']
    if kind == 'post':
        return dict(kind=kind, w=Walker(0), rec=_records(case, seed), n_bins=case['n_bins'], n_cfg=case['n_cfg'])
    make = dict(walk=_prepare_walk, sweep=_prepare_sweep, pol=_prepare_pol, replay=_prepare_replay,
                forward=_prepare_forward, train=_prepare_train, grad=_prepare_grad, retrieve=_prepare_retrieve)[kind]
    return dict(make(case, seed), kind=kind)


# ---------------------------------------------------------------- run


def run(s):
    kind = s['kind']
    if kind == 'walk':
        if s['records'] == 'host':
            r = s['w'].walk(s['cfgs'], s['seed'], out=s['out'])
            return dict(_tallies(r.tallies), **_host_records(r.records))
        if s['records'] == 'device':
            r = s['w'].walk(s['cfgs'], s['seed'], records='device', device_ptr=s['buf'].data_ptr())
            return dict(_tallies(r.tallies), **_device_records(s['buf']))
        return _tallies(s['w'].walk(s['cfgs'], s['seed'], records=None).tallies)
    if kind == 'sweep':
        r = s['graph'].launch(s['seed'])
        return dict(_tallies(r.tallies), **(_device_records(s['buf']) if 'buf' in s else {}))
    if kind == 'pol':
        r = s['w'].walk(s['cfgs'], s['seed'], mode='pol32', out=s['out'])
        return dict(_tallies(r.tallies), **_host_records(r.records, ('stokes_q', 'stokes_u', 'stokes_v')))
    if kind == 'replay':
        r = s['w'].walk(s['cfgs'], s['seed'], mode=s['mode'])
        more = ('stokes_q', 'stokes_u', 'stokes_v') if s['mode'] == 'pol64' else ()
        return dict(_tallies(r.tallies), **_host_records(r.records, more))
    if kind == 'post':
        return post.zenith_brf(s['w'], s['rec'], n_bins=s['n_bins'], n_cfg=s['n_cfg'])
    if kind == 'forward':
        return s['ens'].predict_std(s['x']) if 'ens' in s else s['net'].predict_std(s['x'], half=s['half'])
    if kind == 'train':
        tr = s['tr']
        tr.set_epoch(s['perms'], 1e-3)
        for _ in range(s['steps']):
            tr.run_step()
        return dict(params=tr.params, m=tr.m, v=tr.v, loss=tr.loss)
    if kind == 'grad':
        y = S.mlp_apply(s['x'], s['params'])
        wrt = s['params'] + ([s['x']] if s['x'].requires_grad else [])
        return [y] + list(torch.autograd.grad(y, wrt, s['gy']))
    log_r, brf, spread, spread_r = inverse.surrogate_gn(s['ens'], s['obs'], s['known'], **s['noise'])
    return dict(log_r=log_r, brf=brf, spread=spread, spread_r=spread_r)


# ---------------------------------------------------------------- exact


def _exact_train(c, seed):
    """The epoch's Adam steps in 64 bits, laid out as the engine lays out its parameters: each
    member's W1 (inputs padded to 16), b1, ..., W4, b4, every block on 8 elements."""
    x, t = _inputs(seed, c['batch'] * c['steps']).double(), _targets(seed, c['batch'] * c['steps']).double()
    wl = torch.from_numpy(_loss_weights()).cuda().double()
    out = dict(params=[], m=[], v=[], loss=[])
    for k, perm in enumerate(_perms(c, seed)):
        ps = [p.double().requires_grad_(True) for p in _weights(seed, k)]
        ms, vs = [torch.zeros_like(p) for p in ps], [torch.zeros_like(p) for p in ps]
        total = 0.0
        for i in range(c['steps']):
            rows = torch.from_numpy(perm[i * c['batch']:(i + 1) * c['batch']]).cuda()
            loss = (wl * (_mlp64(x[rows], ps) - t[rows]) ** 2).mean()
            total = float(loss.detach())
            gs = torch.autograd.grad(loss, ps)
            with torch.no_grad():
                for p, g, m, v in zip(ps, gs, ms, vs):
                    m.mul_(0.9).add_(0.1 * g)
                    v.mul_(0.999).add_(0.001 * g * g)
                    p -= 1e-3 * (m / (1 - 0.9 ** (i + 1))) / (torch.sqrt(v / (1 - 0.999 ** (i + 1))) + 1e-8)

        def flat(tensors):
            parts = []
            for j, q in enumerate(tensors):
                q = q.detach()
                if j == 0:
                    q = torch.nn.functional.pad(q, (0, 16 - WIDTHS[0]))
                q = q.reshape(-1)
                parts.append(torch.nn.functional.pad(q, (0, -q.numel() % 8)))
            return torch.cat(parts)
        out['params'].append(flat(ps))
        out['m'].append(flat(ms))
        out['v'].append(flat(vs))
        out['loss'].append(total)
    return dict({k: torch.stack(v) for k, v in out.items() if k != 'loss'},
                loss=torch.tensor(out['loss'], dtype=torch.float64))


def _exact_post(c, seed):
    rec = _records(c, seed)
    n_bins, n_cfg = c['n_bins'], c['n_cfg']
    edges = np.linspace(0., np.pi / 2, n_bins + 1)
    mid = np.diff(edges) / 2. + edges[:-1]
    share = np.sin(mid) * np.cos(mid) / np.sum(np.sin(mid) * np.cos(mid))
    wvn, cond = rec['wvn'].astype(np.float64), rec['condition']
    theta, path, n_scat = (rec[k].astype(np.float64) for k in ('theta_n', 'path_length', 'n_scat'))
    out = dict(midpoints=mid, theta_deg=np.rad2deg(mid), brf=[], hist=[], q_down=[], albedo=[],
               albedo_non_absorbed=[], mean_wavelength=[], mean_n_scat=[], mean_path_length=[], n_cond=[])
    for k in range(n_cfg):
        at = rec['config'] == k
        up = at & (cond == 1)
        hist = np.histogram(theta[up], bins=edges, weights=wvn[up])[0]
        q = wvn[at].sum()
        with np.errstate(invalid='ignore', divide='ignore'):
            out['brf'].append(hist / (q * share))
            out['hist'].append(hist)
            out['q_down'].append(q)
            out['albedo'].append(wvn[up].sum() / q)
            out['albedo_non_absorbed'].append(wvn[at & (cond <= 3)].sum() / q)
            out['mean_wavelength'].append(np.sum(1.0 / wvn[at]) / at.sum())
            out['mean_n_scat'].append(n_scat[at].sum() / at.sum())
            out['mean_path_length'].append(path[at].sum() / at.sum())
            out['n_cond'].append([0.0] + [float(np.sum(at & (cond == j))) for j in range(1, 6)])
    return {k: np.asarray(v, np.float64) for k, v in out.items()}


def exact(case, seed):
    """What `run` returns, in 64 bits.  None for the walks, whose paths hang on every rounding
    of the steps before, and for the retrieval, whose iterations follow the network's own
    rounded outputs."""
    kind = case['kind']
    if kind == 'post':
        return _exact_post(case, seed)
    if kind == 'train':
        return _exact_train(case, seed)
    if kind == 'forward':
        x = _inputs(seed, case['rows']).double()
        ys = [_mlp64(x, [p.double() for p in _weights(seed, k)]) for k in range(case['members'])]
        return ys[0] if case['members'] == 1 else torch.stack(ys)
    if kind == 'grad':
        x = _inputs(seed, case['rows']).double().requires_grad_(case['need_dx'])
        ps = [p.double().requires_grad_(True) for p in _weights(seed, 0)]
        y = _mlp64(x, ps)
        gs = torch.autograd.grad(y, ps + ([x] if case['need_dx'] else []), _targets(seed, case['rows']).double() / case['rows'])
        return [y.detach()] + list(gs)
    return None


# ---------------------------------------------------------------- work


def work(case):
    """Bytes read and written once, and operations: a walk's scatter events (estimated from its
    optics) at OPS_PER_EVENT, a network's multiplies and adds."""
    c, kind = case, case['kind']
    if kind == 'walk':
        ev = _events(c['n'], ssp.co_albedo_synth(c['wvl'], c['r_um']), _tau(c['depth'], c['r_um']))
        return dict(bytes=7888 + (32 * c['n'] if c['records'] != 'none' else 0), flops=OPS_PER_EVENT * ev)
    if kind == 'sweep':
        cfgs = _sweep_configs(c)
        ev = sum(_events(x.n_photon, ssp.co_albedo_synth(x.wvl0, x.rds_snw), x.tau_tot) for x in cfgs)
        return dict(bytes=7888 * len(cfgs) + (32 * sum(x.n_photon for x in cfgs) if c['records'] != 'none' else 0),
                    flops=OPS_PER_EVENT * ev)
    if kind == 'pol':
        # a polarised event also tests about five candidates of the rejection sampler
        ev = _events(c['n'], ssp.co_albedo_synth(c['wvl'], c['re_um']), c['tau'])
        return dict(bytes=7888 + 48 * c['n'], flops=6 * OPS_PER_EVENT * ev)
    if kind == 'replay':
        tau = min(40.0, _tau(c['depth'], c['r_um'])) if c['polarised'] else _tau(c['depth'], c['r_um'])
        ev = _events(c['n'], ssp.co_albedo_synth(c['wvl'], c['r_um']), tau)
        return dict(bytes=7888 + (80 if c['polarised'] else 56) * c['n'],
                    flops=(6 if c['polarised'] else 1) * OPS_PER_EVENT * ev)
    if kind == 'post':
        return dict(bytes=(56 if c['f64'] else 32) * c['n'] + 12 * c['n_bins'] * c['n_cfg'], flops=10 * c['n'])
    if kind == 'forward':
        return dict(bytes=c['members'] * 2 * N_PARAMS + 16 * c['rows'] +
                    c['members'] * c['rows'] * 649 * (2 if c['half'] else 4), flops=c['members'] * c['rows'] * FLOP_ROW)
    if kind == 'train':
        rows = c['members'] * c['batch'] * c['steps']
        return dict(bytes=rows * (16 + 4 * 649) + c['members'] * c['steps'] * 6 * 4 * N_PARAMS, flops=3 * rows * FLOP_ROW)
    if kind == 'grad':
        return dict(bytes=c['rows'] * (16 + 8 * 649) + 8 * N_PARAMS, flops=3 * c['rows'] * FLOP_ROW)
    # a 16-point grid, six iterations and the answer: 18 predictions and seven of value and slope
    return dict(bytes=c['members'] * 2 * N_PARAMS + 16 * 649 * c['n'], flops=(18 + 2 * 7) * c['members'] * c['n'] * FLOP_ROW)
