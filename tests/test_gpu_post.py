"""Post-processing on the device against the reference's own numpy arithmetic
(post_processing.py:73-81 brf; np.histogram binning)."""
import dataclasses

import numpy as np
import pytest

from monte_carlompi_gb300 import _abi, post, ssp
from monte_carlompi_gb300.config import WalkConfig
from tests.conftest import load_golden

pytestmark = pytest.mark.gpu


def reference_brf(wvn, theta, cond, n_bins):
    """post_processing.py:73-81, as the reference computes it."""
    q_down = wvn.sum()
    h = np.histogram(theta[cond == 1], bins=n_bins, range=(0., np.pi / 2), weights=wvn[cond == 1])
    counts = np.histogram(theta[cond == 1], bins=n_bins, range=(0., np.pi / 2))[0]
    midpoints = (np.diff(h[1]) / 2.) + h[1][:-1]
    w = np.sin(midpoints) * np.cos(midpoints) / np.sum(np.sin(midpoints) * np.cos(midpoints))
    return h[0] / (q_down * w), counts, wvn[cond == 1].sum() / q_down, midpoints


def _check(out, rec, n_bins, c=0):
    wvn = rec['wvn'].astype(np.float64)
    theta = rec['theta_n'].astype(np.float64)
    cond = rec['condition']
    brf, counts, albedo, mids = reference_brf(wvn, theta, cond, n_bins)
    assert np.array_equal(out['counts'][c], counts)
    assert np.allclose(out['brf'][c], brf, rtol=1e-9, atol=0)
    assert abs(out['albedo'][c] - albedo) < 1e-9 * albedo
    assert np.array_equal(out['midpoints'], mids)
    q = wvn.sum()
    assert abs(out['albedo_non_absorbed'][c] - wvn[np.isin(cond, (1, 2, 3))].sum() / q) < 1e-9
    assert abs(out['mean_wavelength'][c] - np.mean(1 / wvn)) < 1e-9
    assert abs(out['mean_n_scat'][c] - rec['n_scat'].mean()) < 1e-9
    assert abs(out['mean_path_length'][c] - rec['path_length'].astype(np.float64).mean()) < 1e-6 * abs(
        rec['path_length'].mean()) + 1e-12


@pytest.mark.parametrize('n_bins', [137, 90])
def test_golden_records_match_numpy(walker, n_bins):
    g = load_golden('cfg2')
    rec = np.zeros(g['condition'].size, _abi.RECORD64)
    for k in ('condition', 'n_scat', 'wvn', 'theta_n', 'phi_n', 'path_length', 'snow_depth'):
        rec[k] = g[k]
    out = post.zenith_brf(walker, rec, n_bins)
    _check(out, rec, n_bins)


def test_polarised_records_match_numpy(walker):
    """The polarised walks' records (their leading columns are the HG records') go
    through the same post-processing, FP64 and FP32."""
    from tests.helpers import golden_config, golden_phase, golden_tables
    g = load_golden('pol')
    ice, imp = golden_tables(g)
    walker.set_tables([ice], imp)
    walker.set_phase_matrices([golden_phase(g)])
    for mode in ('pol64', 'pol32'):
        cfg = dataclasses.replace(golden_config(g), n_photon=20000)
        rec = walker.walk([cfg], 9, mode=mode).records
        out = post.zenith_brf(walker, rec, 137)
        _check(out, rec, 137)


def test_walk_records_match_numpy(walker):
    lo, hi = ssp.grid_for(1.55, 0.085)
    walker.set_tables([ssp.synthetic_ice_table(250.0, lo, hi)], ssp.synthetic_impurity_table(lo, hi))
    cfg = WalkConfig(n_photon=200000, wvl0=1.55, half_width=0.085, theta0_deg=60.0,
                     tau_tot=0.02 * ssp.ext_cff_mss_sphere(250.0) * 300.0, lambertian_reflectance=0.5)
    cfg2 = dataclasses.replace(cfg, theta0_deg=0.0, n_photon=50000)
    rec = walker.walk([cfg, cfg2], 3).records
    out = post.zenith_brf(walker, rec, 137)
    _check(out, rec[:200000], 137, c=0)
    _check(out, rec[200000:], 137, c=1)
    assert post.calculate_bins() == 137


def test_bin_edges_follow_numpy():
    """Values on and next to the bin edges land where np.histogram puts them."""
    import torch  # noqa: F401  (GPU context already up via the fixture in other tests)
    from monte_carlompi_gb300.walker import Walker
    n_bins = 90
    edges = np.linspace(0., np.pi / 2, n_bins + 1)
    theta = np.concatenate([edges, np.nextafter(edges, 0), np.nextafter(edges, 4)])
    theta = theta[(theta >= 0) & (theta <= np.pi / 2)]
    rec = np.zeros(theta.size, _abi.RECORD64)
    rec['condition'] = 1
    rec['wvn'] = 0.8
    rec['theta_n'] = theta
    with Walker(0) as w:
        out = post.zenith_brf(w, rec, n_bins)
    ref = np.histogram(theta, bins=n_bins, range=(0., np.pi / 2))[0]
    assert np.array_equal(out['counts'][0], ref)


@pytest.mark.parametrize('n,n_bins,n_cfg,order,dtype', [
    (1, 137, 1, 'sorted', 'RECORD32'), (31, 1, 2, 'sorted', 'RECORD32'), (257, 18, 3, 'mixed', 'RECORD32'),
    (70001, 2048, 5, 'sorted', 'RECORD32P'), (70001, 2049, 5, 'mixed', 'RECORD32'),
    (70001, 137, 300, 'sorted', 'RECORD64'), (70001, 90, 300, 'mixed', 'RECORD64P')])
def test_records_in_any_order_match_numpy(walker, n, n_bins, n_cfg, order, dtype):
    """Block and warp remainders, configs in runs and in no order, bins within and past the
    shared-memory histogram, angles outside [0, pi/2] and undefined, unused conditions."""
    rng = np.random.default_rng(n + n_bins)
    rec = np.zeros(n + 1, getattr(_abi, dtype))[1:]
    rec['condition'] = rng.integers(0, 7, n)
    rec['n_scat'] = rng.integers(0, 2000, n)
    rec['wvn'] = rng.uniform(0.5, 1.2, n)
    rec['theta_n'] = rng.uniform(-0.1, 1.7, n)
    rec['theta_n'][::17] = np.nan
    rec['path_length'] = rng.exponential(0.1, n)
    rec['config'] = rng.integers(0, n_cfg + 1, n)          # one config past the asked ones
    if order == 'sorted':
        rec['config'] = np.sort(rec['config'])
    out = post.zenith_brf(walker, rec, n_bins, n_cfg)
    edges = np.linspace(0., np.pi / 2, n_bins + 1)
    used = (rec['condition'] >= 1) & (rec['condition'] <= 5)
    for c in range(n_cfg):
        at = used & (rec['config'] == c)
        up = at & (rec['condition'] == 1) & np.isfinite(rec['theta_n'])
        theta, wvn = rec['theta_n'][up].astype(np.float64), rec['wvn'].astype(np.float64)
        assert np.array_equal(out['counts'][c], np.histogram(theta, edges)[0])
        assert np.allclose(out['hist'][c], np.histogram(theta, edges, weights=wvn[up])[0], rtol=1e-9, atol=0)
        assert np.array_equal(out['n_cond'][c][1:], [np.sum(at & (rec['condition'] == k)) for k in range(1, 6)])
        assert np.isclose(out['q_down'][c], wvn[at].sum(), rtol=1e-9, atol=0)
        if at.any():
            assert np.isclose(out['mean_wavelength'][c], np.mean(1 / wvn[at]), rtol=1e-12, atol=0)
            assert np.isclose(out['mean_path_length'][c], rec['path_length'][at].astype(np.float64).mean(), rtol=1e-12, atol=0)
            assert out['mean_n_scat'][c] == rec['n_scat'][at].astype(np.int64).sum() / at.sum()


def test_wavelengths_are_correctly_rounded_reciprocals(walker):
    """One record a config: its mean wavelength is 1 / wvn to the last bit, also where the quotient
    lies next to the middle between two doubles (2 - k 2^-52, k odd) and in the least and largest
    binades."""
    x = np.concatenate([(2.0 - np.arange(1, 4001, 2) * 2.0 ** -52) * s for s in (1.0, 0.25, 2.0 ** -20)] +
                       [np.random.default_rng(3).uniform(0.3, 3.0, 4000), [1e-300, 2.0 ** -960, 2.0 ** 900, 0.5, 1.0, 3.0]])
    rec = np.zeros(x.size, _abi.RECORD64)
    rec['condition'], rec['wvn'], rec['config'] = 2, x, np.arange(x.size)
    out = post.zenith_brf(walker, rec, 8, x.size)
    assert np.array_equal(out['mean_wavelength'], 1 / x)
