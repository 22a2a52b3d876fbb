"""Blackbody ring records: a point's value has the rounding that the tiles give it, whatever it is batched with."""
import numpy as np
import pytest

from gpu_ppm_b200 import _abi, synth
from gpu_ppm_b200.engine import Engine

pytestmark = pytest.mark.gpu


def _engine():
    e = Engine()
    e.load_lensing(synth.lensing("std"))
    return e


@pytest.mark.parametrize("precision", [_abi.PREC_FP64, _abi.PREC_FP32])
def test_light_curve_bits_do_not_depend_on_the_batch(monkeypatch, precision):
    """Small caps of a fast star, E / kT around 1 at their points: rings of few elements, of which several nodes share a
    warp (how many depends on the records of the batch)."""
    monkeypatch.setenv("PPM_RECORDS", "1")
    e = _engine()
    g = e.add_energy_grid(np.array([0.36, 0.37, 0.38, 0.39]))

    def light_curve(theta, angle, n_side):
        return synth.params(mass_msun=1.0, r_eq_km=16.0, spin_hz=700.0, inclination_rad=1.3, distance_kpc=0.2,
                            spots=[synth.spot(theta, 0.2, angle, kT_keV=0.35)], atmosphere=_abi.ATM_BLACKBODY,
                            beaming=0, n_side=n_side, n_bins=64, n_gl=2, n_fine=192, energy_grid=g,
                            precision=precision)

    caps = [light_curve(1.2 + 0.02 * k, 0.08, 16) for k in range(20)]
    out = []
    for n_fill in (1, 2):
        flux, _, infos = e.profile_batch(caps + [light_curve(1.4, 0.45, 110)] * n_fill, want_counts=False)
        assert 1.35 * 148 < sum(i.n_rings for i in infos) < 4 * 148
        out.append(flux[:20])
    for a, b in zip(*out):
        assert a.any() and np.array_equal(a, b)
    e.close()


@pytest.mark.parametrize("precision", [_abi.PREC_FP64, _abi.PREC_FP32])
@pytest.mark.parametrize("n_e", [5, 64, 65, 300])
def test_one_point_has_the_bits_of_the_tiles(monkeypatch, n_e, precision):
    """One term a bin, so that no order of summation shows: the phase fraction, the lerps and the Planck factor round as
    from tiles."""
    out = []
    for records in ("1", "0"):
        monkeypatch.setenv("PPM_RECORDS", records)
        e = _engine()
        g = e.add_energy_grid(synth.energy_grid(n_e, 0.05, 15.0))
        one = synth.params(mass_msun=1.4, r_eq_km=12.0, spin_hz=400.0, inclination_rad=1.1, distance_kpc=0.2,
                           spots=[synth.spot(0.9, 0.1, 0.1, kT_keV=0.3)], atmosphere=_abi.ATM_BLACKBODY, beaming=1,
                           n_side=32, n_bins=200, n_gl=0, n_fine=150, energy_grid=g, precision=precision)
        one.spots[0].kind = _abi.SPOT_POINT
        out.append(e.profile(one, want_counts=False))
        e.close()
    assert out[0][2].as_dict() == out[1][2].as_dict() and out[0][2].n_points > 0
    assert np.array_equal(out[0][0], out[1][0])
