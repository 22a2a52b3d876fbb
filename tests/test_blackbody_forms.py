"""The two forms of a blackbody group, tiles and ring records, give the same values: with memory for all of the records'
node sums, for some (the others are added to the flux pool atomically) and for none.

Tolerance: FP64 terms round alike in both forms and are positive, their sums are compensated: 1e-12.  In FP32 the forms
fuse products and sums differently, half a unit of 2^-23 at E z / kT, which the exponential magnifies by up to that
number, 60 here: 2e-5."""
import numpy as np
import pytest

from gpu_ppm_b200 import _abi, synth
from gpu_ppm_b200.engine import Engine
from tests.errors import max_rel

pytestmark = pytest.mark.gpu

N_SIDE, N_BINS, N_GL, N_FINE = 20, 9, 3, 54


def _run(monkeypatch, records, budget, E, precision):
    monkeypatch.setenv("PPM_RECORDS", records)
    e = Engine(memory_budget=budget)
    e.load_lensing(synth.lensing("std"))
    g = e.add_energy_grid(E)
    p = synth.params(mass_msun=1.4, r_eq_km=12.0, spin_hz=400.0, inclination_rad=1.1, distance_kpc=0.2,
                     spots=[synth.spot(1.0, 0.1, 0.5, kT_keV=0.3), synth.spot(2.2, 3.0, 0.4, 2.2, 3.1, 0.2, kT_keV=0.25)],
                     atmosphere=_abi.ATM_BLACKBODY, beaming=1, n_side=N_SIDE, n_bins=N_BINS, n_gl=N_GL, n_fine=N_FINE,
                     energy_grid=g, precision=precision)
    flux, _, info = e.profile(p, want_counts=False)
    again, _, _ = e.profile(p, want_counts=False)
    e.close()
    assert max_rel(again, flux) < 1e-15
    return flux, info.as_dict()


@pytest.mark.parametrize("precision", [_abi.PREC_FP64, _abi.PREC_FP32])
@pytest.mark.parametrize("n_e", [1, 4, 5, 33, 64, 65, 129, 300])
def test_same_values_with_all_some_and_none_of_the_node_sums(monkeypatch, n_e, precision):
    E = synth.energy_grid(n_e, 0.1, 12.0) if n_e > 1 else np.array([1.0])
    tol = 1e-12 if precision == _abi.PREC_FP64 else 2e-5
    tiles, info = _run(monkeypatch, "0", 0, E, precision)
    # the records of one profile of this size take 1 MiB of the eighth of the budget; a record's node sums:
    each = 4 * ((n_e * N_BINS * N_GL * 2 + 63) // 64 * 64)
    some = 1 << (12 * each).bit_length() - 1
    assert 0 < some // each < info["n_rings"]
    for left in (None, some, 0):
        flux, rec_info = _run(monkeypatch, "1", 0 if left is None else 8 * ((1 << 20) + left), E, precision)
        assert rec_info == info, left
        assert max_rel(flux, tiles) < tol, left
