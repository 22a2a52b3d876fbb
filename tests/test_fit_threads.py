"""Fit statistics of one batch from several threads and streams at once: every call returns the batch's statistics
against its own observed data."""
import ctypes
import threading

import numpy as np
import pytest

from gpu_ppm_b200 import _abi, synth


@pytest.mark.gpu
def test_fits_of_one_batch_from_two_threads():
    import torch

    from gpu_ppm_b200.engine import Engine

    e = Engine()
    e.load_lensing(synth.lensing("std"))
    e.load_nsx(synth.nsx("v171019", seed=0))
    E = synth.energy_grid(24, 0.2, 12.0)
    g = e.add_energy_grid(E)
    r = e.add_response(g, synth.response(300, 24, E, seed=0))
    plist, _ = synth.draw_prior(400, seed=7, lens_u=(0.3, 0.5), n_side=4, n_bins=64, energy_grid=g, response=r,
                                fold=_abi.FOLD_FP64)
    rng = np.random.default_rng(3)
    ids = [e.add_observed(r, 64, rng.poisson(3.0 + k, size=(300, 64)).astype(float)) for k in range(2)]
    batch = e.batch(plist)
    batch.launch()
    batch.collect(want_counts=False)
    streams = [torch.cuda.Stream() for _ in ids]

    def fit(k):
        out = (_abi.Fit * len(plist))()
        _abi.check(_abi.lib().ppm_batch_fit(e.h, batch.h, ids[k], out, ctypes.c_void_p(streams[k].cuda_stream)))
        return bytes(out)

    want = [fit(k) for k in range(2)]
    wrong = [0, 0]

    def work(k):
        for _ in range(300):
            wrong[k] += fit(k) != want[k]

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert wrong == [0, 0] and [fit(k) for k in range(2)] == want
    batch.close()
    e.close()
