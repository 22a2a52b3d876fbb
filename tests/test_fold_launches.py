"""The tensor-core fold at the edges of its loads, conversion and launches:
energies that do not fill a chunk or align a row, rows and channels around the
tiles, values outside FP32's normal range, and more folds than one launch takes.

Tolerance: each operand keeps 16 bits (2^-17 relative each, 2^-18 for the
product left out) and up to 300 products are summed in FP32 (300 x 6e-8):
1e-4 of the sum of magnitudes, and FP32's smallest normal number per term."""
import numpy as np
import pytest

import oracle
from gpu_ppm_b200 import _abi, synth

pytestmark = pytest.mark.gpu


def _engine():
    from gpu_ppm_b200.engine import Engine

    e = Engine()
    e.load_lensing(synth.lensing("std"))
    e.load_nsx(synth.nsx("v171019", seed=0))
    return e


@pytest.mark.parametrize("n_e", [2, 27, 32, 33, 299, 300])
@pytest.mark.parametrize("n_ch,n_bins", [(1, 1), (33, 129), (257, 64)])
def test_fold_edges_and_values(n_e, n_ch, n_bins):
    e = _engine()
    rng = np.random.default_rng(n_e * n_ch)
    E = synth.energy_grid(n_e, 0.2, 12.0)
    rsp = rng.uniform(0.0, 1.0, size=(n_ch, n_e))
    r = e.add_response(e.add_energy_grid(E), rsp)
    flux = rng.uniform(-1.0, 1.0, size=(n_bins, n_e)) * 10.0 ** rng.integers(-6, 6, size=(n_bins, 1))
    flux[::5] = 0.0
    flux[1::7] *= 1e-40   # below FP32's normal numbers
    flux[2::7, ::2] = 5e-320
    flux[3::7] = rng.uniform(1e30, 1e33, size=flux[3::7].shape)
    got = np.asarray(e.fold(r, flux, 2.0 / n_bins, _abi.FOLD_BF16X3)).reshape(n_ch, n_bins)
    want = oracle.fold(rsp, flux, 2.0)
    bound = 1e-4 * oracle.fold(rsp, np.abs(flux), 2.0) + 1.2e-38 * n_e * 2.0 / n_bins
    assert np.all(np.abs(got - want) <= bound)
    if n_bins > 1:  # a row that is not finite stays alone
        flux[4, 0] = np.inf
        bad = np.asarray(e.fold(r, flux, 2.0 / n_bins, _abi.FOLD_BF16X3)).reshape(n_ch, n_bins)
        keep = np.arange(n_bins) != 4
        assert np.array_equal(bad[:, keep], got[:, keep])
        assert not np.isfinite(bad[:, 4]).any()
    e.close()


@pytest.mark.parametrize("n_folds", [2, 16, 17])
def test_folds_of_a_batch_share_launches(n_folds):
    e = _engine()
    E = synth.energy_grid(40, 0.2, 12.0)
    g = e.add_energy_grid(E)
    rng = np.random.default_rng(n_folds)
    plist, chs = [], []
    for k in range(n_folds):
        n_ch = int(rng.integers(1, 300))
        r = e.add_response(g, rng.uniform(0.0, 1.0, size=(n_ch, 40)))
        plist += synth.draw_prior(2, seed=k, lens_u=(0.3, 0.5), n_side=4, n_bins=8 if k % 3 else 130, energy_grid=g,
                                  response=r, fold=_abi.FOLD_BF16X3)[0]
        chs += [n_ch, n_ch]
    batch = e.batch(plist)
    batch.launch()
    flux, counts, _ = batch.collect(want_flux=True, want_counts=True)
    f0 = c0 = 0
    for p, n_ch in zip(plist, chs):
        f = np.asarray(flux[f0:f0 + p.n_bins * 40]).reshape(p.n_bins, 40)
        alone = np.asarray(e.fold(p.response, f, p.exposure_s / p.n_bins, _abi.FOLD_BF16X3)).ravel()
        assert np.array_equal(counts[c0:c0 + n_ch * p.n_bins], alone)
        f0 += p.n_bins * 40
        c0 += n_ch * p.n_bins
    batch.close()
    e.close()
