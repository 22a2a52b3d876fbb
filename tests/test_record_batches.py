"""Batches of many profiles from ring records: a ring's job finds its profile and spot among more profiles than a CTA
has threads, and a profile's flux is summed from its own list of records."""
import numpy as np
import pytest

from gpu_ppm_b200 import _abi, synth
from tests.errors import max_rel

pytestmark = pytest.mark.gpu


def _spectra(g, n):
    """Blackbody spectra: one or two spots, caps of few and many rings, point sources, caps smaller than a ring."""
    rng = np.random.default_rng(n)
    out = []
    for k in range(n):
        spots = [synth.spot(float(rng.uniform(0.2, 2.9)), 0.1 * k, float(rng.choice([0.001, 0.05, 0.4])), kT_keV=0.3)]
        if k % 3 == 0:
            spots.append(synth.spot(2.0, 3.0, 0.2, kT_keV=0.2))
        p = synth.params(mass_msun=1.4, r_eq_km=12.0, spin_hz=400.0, inclination_rad=1.1, distance_kpc=0.2, spots=spots,
                         atmosphere=_abi.ATM_BLACKBODY, beaming=0, n_side=4 + k % 9, n_bins=3 + k % 4, n_gl=k % 3,
                         n_fine=40, energy_grid=g, precision=_abi.PREC_FP64)
        if k % 4 == 1:
            p.spots[0].kind = _abi.SPOT_POINT
        if k % 6 == 3:
            p.spots[1].kind = _abi.SPOT_POINT
        out.append(p)
    return out


@pytest.mark.parametrize("n,n_e", [(2, 33), (255, 5), (256, 7), (257, 6), (700, 40)])
def test_profiles_of_a_batch(monkeypatch, n, n_e):
    from gpu_ppm_b200.engine import Engine

    monkeypatch.setenv("PPM_RECORDS", "1")
    e = Engine()
    e.load_lensing(synth.lensing("std"))
    g = e.add_energy_grid(synth.energy_grid(n_e, 0.1, 12.0))
    plist = _spectra(g, n)
    flux, _, infos = e.profile_batch(plist, want_counts=False)
    for k in sorted({n // 2, n - 2, n - 1} | set(range(0, n, max(1, n // 40)))):
        one, _, info = e.profile(plist[k], want_counts=False)
        assert infos[k].as_dict() == info.as_dict(), k
        assert max_rel(flux[k], one) < 1e-12, k  # FP64 sums of another order
    e.close()


def test_more_profiles_than_a_grid_dimension_holds(monkeypatch):
    """65 540 profiles, of which the ring window leaves five with rings, the last one among them."""
    from gpu_ppm_b200.engine import Engine

    monkeypatch.setenv("PPM_RECORDS", "1")
    e = Engine(max_batch=70000)
    e.load_lensing(synth.lensing("std"))
    g = e.add_energy_grid(synth.energy_grid(5, 0.1, 12.0))
    # one cap around the pole (rings 1 and 2 of 15), the others around the equator
    polar, far = [synth.params(mass_msun=1.4, r_eq_km=12.0, spin_hz=400.0, inclination_rad=1.1, distance_kpc=0.2,
                               spots=[synth.spot(t, 0.0, 0.4, kT_keV=0.3)], atmosphere=_abi.ATM_BLACKBODY, beaming=0,
                               n_side=4, n_bins=2, n_gl=0, n_fine=8, energy_grid=g, precision=_abi.PREC_FP64)
                  for t in (0.1, 1.6)]
    plist = [far] * 65540
    own = [0, 1, 40000, 65535, 65539]
    for k in own:
        plist[k] = polar
    batch = e.batch(plist, rings=(1, 3))
    batch.launch()
    flux, _, infos = batch.collect(want_flux=True, want_counts=False)
    batch.close()
    one, _, info = e.profile_rings(polar, 1, 3, want_counts=False)
    e.close()
    flux = np.asarray(flux).reshape(len(plist), -1)
    assert info.n_points > 0 and one.any()
    for k in own:
        assert infos[k].as_dict() == info.as_dict()
        assert max_rel(flux[k], one.ravel()) < 1e-12
    assert not np.delete(flux, own, axis=0).any()
