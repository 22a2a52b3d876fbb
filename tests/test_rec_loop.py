"""The loop that hands chunks and phase nodes to the warp sets of a ring-record CTA (rec_loop, csrc/rec_loop.cuh).

On the host: tests/rec_loop_check.cpp runs the loop's own source on host threads that read what a set's leader hands
out as late as its barriers allow.  On the GPU: warp sets of several warps with more chunks than all slots hold, so
that every set reloads its slots, against the path over tiles: the same bits."""
import os
import subprocess

import numpy as np
import pytest

from gpu_ppm_b200 import build as B
from gpu_ppm_b200 import synth

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_hand_out_with_late_readers(tmp_path):
    cuda_include = os.path.join(os.path.dirname(os.path.dirname(B.NVCC)), "include")
    if not os.path.exists(os.path.join(cuda_include, "cuda_runtime.h")):
        pytest.skip("CUDA headers not available")
    exe = tmp_path / "rec_loop_check"
    subprocess.run(["g++", "-std=c++20", "-O1", "-w", "-pthread", "-I", os.path.join(ROOT, "include"), "-I", B.CSRC,
                    "-I", cuda_include, os.path.join(HERE, "rec_loop_check.cpp"), "-o", str(exe)], check=True,
                   capture_output=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300).stdout.split()
    assert out == ["8", "0"]


@pytest.mark.gpu
@pytest.mark.parametrize("n_e,lo,hi", [(600, 0.2, 12.0), (400, 0.02, 60.0)])
def test_sets_of_several_warps_reload_their_slots(monkeypatch, n_e, lo, hi):
    from gpu_ppm_b200.engine import Engine

    E = synth.energy_grid(n_e, lo, hi)
    out = []
    for splits in ("1", None):  # tiles, records
        if splits:
            monkeypatch.setenv("PPM_SPLITS", splits)
        else:
            monkeypatch.delenv("PPM_SPLITS")
        e = Engine()
        e.load_lensing(synth.lensing("std"))
        e.load_nsx(synth.nsx("v171019", seed=2))
        g = e.add_energy_grid(E)
        plist = [synth.config2_params(g, -1, n_side=64 + 3 * k, n_bins=16) for k in range(10)]
        for k, p in enumerate(plist):
            p.n_spots = 1
            p.spots[0] = synth.params(spots=[synth.spot(0.8 + 0.1 * k, 0.3 * k, 0.9, logT=5.9)]).spots[0]
        flux, _, infos = e.profile_batch(plist, want_counts=False)
        out.append((flux, [i.as_dict() for i in infos]))
        e.close()
    assert out[0][1] == out[1][1]
    assert sum(i["n_rings"] for i in out[0][1]) > 4 * 148
    for a, b in zip(out[0][0], out[1][0]):
        assert np.array_equal(a, b)
