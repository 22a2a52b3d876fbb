"""Blackbody ring records: a point's value has the rounding that the tiles give it, whatever it is batched with."""
import numpy as np
import pytest

from gpu_ppm_b200 import _abi, synth
from gpu_ppm_b200.engine import Engine

pytestmark = pytest.mark.gpu


def _engine(budget=0):
    e = Engine(memory_budget=budget)
    e.load_lensing(synth.lensing("std"))
    return e


@pytest.mark.parametrize("precision", [_abi.PREC_FP64, _abi.PREC_FP32])
def test_light_curve_bits_do_not_depend_on_the_batch(precision):
    """Small caps of a fast star, E / kT around 1 at their points: rings of few elements, of which several nodes share a
    warp (how many depends on the records of the batch)."""
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
