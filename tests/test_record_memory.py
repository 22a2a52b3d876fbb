"""Device memory of ring records: batch objects that exist together share an eighth of the engine's memory budget, the
ones beyond that run from tiles, with the same bits; a destroyed batch gives its share back."""
import numpy as np
import pytest

from gpu_ppm_b200 import synth
from gpu_ppm_b200.engine import Engine

pytestmark = pytest.mark.gpu


def test_batches_share_the_engines_ring_memory():
    import torch

    e = Engine(memory_budget=2 << 30)
    e.load_lensing(synth.lensing("std"))
    e.load_nsx(synth.nsx("v171019", seed=0))
    g = e.add_energy_grid(synth.energy_grid(300, 0.2, 12.0))
    p = synth.config2_params(g, -1, n_side=256, n_bins=64)
    p.n_gl = 2
    e.profile(p, want_counts=False)
    torch.cuda.synchronize()

    def make(n):
        before = torch.cuda.mem_get_info()[0]
        batches = [e.batch([p]) for _ in range(n)]
        took = before - torch.cuda.mem_get_info()[0]
        flux = []
        for b in batches:
            b.launch()
            flux.append(np.array(b.collect(want_flux=True, want_counts=False)[0]))
            b.close()
        return took, flux

    # 160 MB of records and sums each: the first has its own, the others what is left of 256 MB; and each its outputs
    # and tiles, a few MB
    took, flux = make(10)
    assert took < (256 << 20) + 10 * (16 << 20)
    for f in flux[1:]:
        assert np.array_equal(f, flux[0])
    assert np.array_equal(make(1)[1][0], flux[0])
    e.close()
