"""Blackbody groups from ring records (integrand_bb_rec_kernel): energies on every side of its lane and pass
boundaries, rings of few and many elements, both arithmetics, two spots, against the oracle.  FP64 differs from the
oracle by rounding alone (sums of up to 1e6 terms of relative error 2^-52 each: below 1e-9); FP32 evaluates in 24 bits."""
import numpy as np
import pytest

import oracle
from gpu_ppm_b200 import _abi, synth
from gpu_ppm_b200.engine import Engine
from tests.errors import max_rel

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    e = Engine()
    e.load_lensing(synth.lensing("std"))
    e.ora = oracle.Oracle(synth.lensing("std"))
    yield e
    e.close()


def _params(g, precision, n_side, n_bins, n_gl, spots, beaming):
    return synth.params(mass_msun=1.4, r_eq_km=12.0, spin_hz=400.0, inclination_rad=1.1, distance_kpc=0.2, spots=spots,
                        atmosphere=_abi.ATM_BLACKBODY, beaming=beaming, n_side=n_side, n_bins=n_bins, n_gl=n_gl,
                        n_fine=6 * n_bins, energy_grid=g, precision=precision)


@pytest.mark.parametrize("precision", [_abi.PREC_FP64, _abi.PREC_FP32])
@pytest.mark.parametrize("n_e", [5, 8, 9, 16, 17, 32, 33, 64, 65, 128, 129, 257, 300])
def test_energies(eng, n_e, precision):
    E = synth.energy_grid(n_e, 0.05, 15.0)
    g = eng.add_energy_grid(E)
    spots = [synth.spot(1.0, 0.1, 0.5, kT_keV=0.3), synth.spot(2.2, 3.0, 0.4, 2.2, 3.1, 0.2, kT_keV=0.15)]
    plist = [_params(g, precision, 13, 9, 1 + n_e % 3, spots, n_e % 3), _params(g, precision, 41, 5, 2, spots[:1], 0)]
    flux, _, infos = eng.profile_batch(plist, want_counts=False)
    for k, p in enumerate(plist):
        one, _, info = eng.profile(p, want_counts=False)
        ref, oinfo = eng.ora.profile(p, E)
        assert info.as_dict() == infos[k].as_dict() and info.n_points == oinfo.n_points
        assert info.n_active == oinfo.n_active
        assert max_rel(one, ref) < (1e-9 if precision == _abi.PREC_FP64 else 1e-4), n_e
        assert max_rel(flux[k], one) < 1e-12


@pytest.mark.parametrize("precision", [_abi.PREC_FP64, _abi.PREC_FP32])
@pytest.mark.parametrize("n_e,n_gl", [(1, 0), (1, 2), (3, 0), (4, 3)])
def test_light_curves_of_many_rings(eng, n_e, n_gl, precision):
    """Few energies: 229 rings or more on 148 SMs run from ring records, with up to 600 elements a ring and, at the
    pole and the rim, fewer than 16 (several nodes at a time)."""
    E = np.linspace(0.7, 2.0, n_e)
    g = eng.add_energy_grid(E)
    p = _params(g, precision, 150, 11, n_gl, [synth.spot(0.9, 0.2, 1.2, kT_keV=0.35)], 1)
    flux, _, info = eng.profile(p, want_counts=False)
    ref, oinfo = eng.ora.profile(p, E)
    assert info.n_points == oinfo.n_points and info.n_active == oinfo.n_active
    assert max_rel(flux, ref) < (1e-9 if precision == _abi.PREC_FP64 else 1e-4)
