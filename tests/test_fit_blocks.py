"""Fit statistics at the sizes where a profile's entries move from one block to
the next, and to the largest number of blocks, against the restatements of
cal_chi2 and the Poisson log-likelihood.

Tolerance: 1e-10 relative (both sides FP64; only the summation order differs:
200 000 terms x 1.1e-16, and the log-likelihood's terms cancel by less than 1e3)."""
import numpy as np
import pytest

import oracle
from gpu_ppm_b200 import _abi, synth


@pytest.mark.gpu
@pytest.mark.parametrize("n_ch,n_bins", [(1, 1), (5, 51), (32, 32), (1025, 1), (241, 17), (512, 64), (331, 99), (513, 384)])
def test_fit_statistics_across_block_counts(n_ch, n_bins):
    from gpu_ppm_b200.engine import Engine

    e = Engine()
    e.load_lensing(synth.lensing("std"))
    e.load_nsx(synth.nsx("v171019", seed=0))
    E = synth.energy_grid(24, 0.2, 12.0)
    g = e.add_energy_grid(E)
    r = e.add_response(g, synth.response(n_ch, 24, E, seed=0))
    plist, _ = synth.draw_prior(3, seed=7, lens_u=(0.3, 0.5), n_side=4, n_bins=n_bins, energy_grid=g, response=r,
                                fold=_abi.FOLD_FP64)
    rng = np.random.default_rng(n_ch)
    obs = rng.poisson(3.0, size=(n_ch, n_bins)).astype(float)
    oid = e.add_observed(r, n_bins, obs)
    batch = e.batch(plist)
    batch.launch()
    _, counts, _ = batch.collect(want_counts=True)
    first = batch.fit(oid)
    assert repr(first) == repr(batch.fit(oid))  # the counters are back at zero
    n_el = n_ch * n_bins
    for k in range(len(plist)):
        m = counts[k * n_el:(k + 1) * n_el]
        d = obs.ravel()
        assert first[k]["model_total"] == pytest.approx(m.sum(), rel=1e-12)
        assert first[k]["n_zero_model"] == int((m <= 0).sum())
        if m.sum() <= 0:
            continue
        assert first[k]["chi2"] == pytest.approx(oracle.cal_chi2(d, m), rel=1e-10)
        ll = oracle.poisson_loglike(d, m)
        assert first[k]["loglike"] == (ll if np.isinf(ll) else pytest.approx(ll, rel=1e-10))
    batch.close()
    e.close()
