"""The home-cell path of small batches (ring records: ring_kernel, integrand_nsx_rec_kernel, sum_parts_kernel)
against the path over tiles, which a small memory budget or PPM_SPLITS=1 selects: the same bits, for every
slot count of the kernels, interpolator and table end, with all, some or none of the node sums in memory."""
import numpy as np
import pytest

import oracle
from gpu_ppm_b200 import _abi, synth
from gpu_ppm_b200.engine import Engine
from tests.errors import max_rel

pytestmark = pytest.mark.gpu

# energies per NSX cell (0.02 dex): 1, 2, 3, 4, 7, 14; two warps of cells; a descending grid; one energy
GRIDS = {
    "maxe1": synth.energy_grid(60, 0.2, 12.0), "maxe2": synth.energy_grid(128, 0.2, 12.0),
    "maxe3": synth.energy_grid(211, 0.2, 12.0), "maxe4": synth.energy_grid(300, 0.2, 12.0),
    "maxe8": synth.energy_grid(600, 0.2, 12.0), "maxe16": synth.energy_grid(1200, 0.2, 12.0),
    "two_warps": synth.energy_grid(400, 0.02, 60.0), "descending": synth.energy_grid(90, 0.2, 12.0)[::-1].copy(),
    "one": np.array([1.0]),
}


def _profiles(g, interp, n_gl):
    """A ring and a crescent, a disk of every azimuth with odd sizes, a point source."""
    a = synth.config2_params(g, -1, n_side=21, n_bins=13)
    b = synth.config2_params(g, -1, n_side=40, n_bins=7)
    b.n_spots = 1
    b.spots[0] = synth.params(spots=[synth.spot(0.0, 0.0, 0.9, logT=5.85)]).spots[0]
    c = synth.config2_params(g, -1, n_side=21, n_bins=13)
    c.spots[1].kind = _abi.SPOT_POINT
    for p in (a, b, c):
        p.interp = interp
        p.n_gl = n_gl
        p.n_fine = 6 * p.n_bins
    return [a, b, c]


def _run(E, interp, n_gl, nsx, budget, monkeypatch, splits=None):
    if splits:
        monkeypatch.setenv("PPM_SPLITS", splits)
    else:
        monkeypatch.delenv("PPM_SPLITS", raising=False)
    e = Engine(memory_budget=budget)
    try:
        e.load_lensing(synth.lensing("std"))
        e.load_nsx(nsx)
        g = e.add_energy_grid(E)
        plist = _profiles(g, interp, n_gl)
        one = [e.profile(p, want_counts=False) for p in plist]
        flux, _, infos = e.profile_batch(plist, want_counts=False)
        return plist, [f for f, _, _ in one], [i.as_dict() for _, _, i in one], flux, [i.as_dict() for i in infos]
    finally:
        e.close()


@pytest.mark.parametrize("grid", GRIDS)
def test_same_bits_as_tiles(monkeypatch, grid):
    nsx = synth.nsx("v171019", seed=2)
    k = list(GRIDS).index(grid)
    interp, n_gl = (3, 0, 1, 2, 4)[k % 5], (2, 1, 3)[k % 3]
    plist, tiles, tile_info, _, _ = _run(GRIDS[grid], interp, n_gl, nsx, 0, monkeypatch, splits="1")
    # 8.5 MB: the records of a small batch fit, its node sums only in part; 4 MB: not even the records
    for budget in (0, 17 << 19, 4 << 20):
        _, one, info, flux, infos = _run(GRIDS[grid], interp, n_gl, nsx, budget, monkeypatch)
        for q in range(len(plist)):
            assert np.array_equal(one[q], tiles[q]), (budget, q, max_rel(one[q], tiles[q]))
            assert np.array_equal(flux[q], tiles[q]), (budget, q)
            assert info[q] == tile_info[q] and infos[q] == tile_info[q], (budget, q)
    ref, oinfo = oracle.Oracle(synth.lensing("std"), nsx).profile(plist[0], GRIDS[grid])
    assert tile_info[0]["n_points"] == oinfo.n_points and max_rel(tiles[0], ref) < 1e-4


@pytest.mark.parametrize("axis", [(0.6, 1.4), (-0.3, 0.5)])
def test_table_ends_and_even_mu(monkeypatch, axis):
    """Energies with large flux past either end of the logEkT axis, even mu count (padded slice rows)."""
    nsx = synth.nsx("v171019", seed=1, n_mu=66, dims={"n_logEkT": 41, "logEkT": axis})
    for interp in range(5):
        E = GRIDS["maxe4"]
        plist, tiles, tile_info, _, _ = _run(E, interp, 2, nsx, 0, monkeypatch, splits="1")
        _, one, info, flux, _ = _run(E, interp, 2, nsx, 0, monkeypatch)
        for q in range(len(plist)):
            assert np.array_equal(one[q], tiles[q]) and np.array_equal(flux[q], tiles[q]), (interp, q)
            assert info[q] == tile_info[q]
        ref, oinfo = oracle.Oracle(synth.lensing("std"), nsx).profile(plist[0], E)
        assert info[0]["n_points"] == oinfo.n_points and info[0]["n_clamped"] > 0
        assert max_rel(one[0], ref) < 1e-4
