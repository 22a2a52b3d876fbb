"""The tile form of the home-cell kernel in its two block sizes (three small blocks an SM where tiles are small, two of
ten warps else) and with nodes split over tiles: the bits of the ring records, at grids of one warp a set and of two."""
import numpy as np
import pytest

import oracle
from gpu_ppm_b200 import synth
from gpu_ppm_b200.engine import Engine
from tests.errors import max_rel

pytestmark = pytest.mark.gpu


def _batch(monkeypatch, records, E, shapes):
    monkeypatch.setenv("PPM_RECORDS", records)
    e = Engine()
    e.load_lensing(synth.lensing("std"))
    e.load_nsx(synth.nsx("v171019", seed=2))
    g = e.add_energy_grid(E)
    plist = []
    for k, (n_side, n_bins, angle) in enumerate(shapes):
        p = synth.config2_params(g, -1, n_side=n_side, n_bins=n_bins)
        p.n_gl, p.n_fine, p.n_spots = 1 + k % 2, 6 * n_bins, 1
        p.spots[0] = synth.params(spots=[synth.spot(0.7 + 0.03 * k, 0.1 + k % 6, angle, logT=5.9)]).spots[0]
        plist.append(p)
    flux, _, infos = e.profile_batch(plist, want_counts=False)
    e.close()
    return plist, flux, [i.as_dict() for i in infos]


# (N_side, bins, radius) of the profiles: more than two tiles an SM with few points each; two profiles whose
# nodes are split; 30 large ones
SHAPES = {"small": [(12 + k % 7, 8 + k % 3, 0.25) for k in range(50)], "split": [(40, 24, 0.5), (31, 24, 0.3)],
          "large": [(48, 24, 0.5)] * 30}


@pytest.mark.parametrize("n_e,lo,hi", [(60, 0.2, 12.0), (300, 0.2, 12.0), (600, 0.2, 12.0), (400, 0.02, 60.0)])
@pytest.mark.parametrize("shape", SHAPES)
def test_same_bits_as_records(monkeypatch, n_e, lo, hi, shape):
    E = synth.energy_grid(n_e, lo, hi)
    plist, tiles, info = _batch(monkeypatch, "0", E, SHAPES[shape])
    _, recs, rec_info = _batch(monkeypatch, "1", E, SHAPES[shape])
    assert info == rec_info
    for a, b in zip(tiles, recs):
        assert np.array_equal(a, b)
    ref, oinfo = oracle.Oracle(synth.lensing("std"), synth.nsx("v171019", seed=2)).profile(plist[0], E)
    assert info[0]["n_points"] == oinfo.n_points and max_rel(tiles[0], ref) < 1e-4
