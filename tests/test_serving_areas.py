"""Served batches whose memory comes from the stream slots' areas, from the areas and the stream-ordered pool, or mostly
from the pool: the same bits as the profiles alone.  The areas are shares of the memory budget."""
import numpy as np
import pytest

from gpu_ppm_b200 import synth
from gpu_ppm_b200.engine import Engine
from tests.test_serving import mixed_requests, submit_all

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("budget,n_streams", [(0, 3), (400 << 20, 1), (64 << 20, 2), (20 << 20, 3)])
def test_served_bits_with_areas_of_any_size(budget, n_streams):
    e = Engine(n_streams=n_streams, memory_budget=budget)
    e.load_lensing(synth.lensing("wide"))
    e.load_nsx(synth.nsx("v171019", seed=0))
    grids = {}
    for n in (128, 300):
        E = synth.energy_grid(n, 0.2, 12.0)
        g = e.add_energy_grid(E)
        grids[n] = (g, {ch: e.add_response(g, synth.response(ch, 1000, E, seed=0)) for ch in (300, 1500)})
    reqs = mixed_requests(grids, 40, seed=5)
    for _ in range(2):  # the second time from areas that were used
        for p, (flux, counts) in zip(reqs, submit_all(e, reqs)):
            one, one_counts, _ = e.profile(p)
            assert np.array_equal(flux, one) and np.array_equal(counts, one_counts)
    e.close()
