"""The row-owner kernel on lattices that leave warps without rows, slices partly
filled, and sites without neighbours, in whole waves of 8-vector CTAs and a
remainder: against the sliced-ELL kernel (kernel_config 13) and FP64."""
import numpy as np
import pytest

import helpers
import nise_2017_b200 as nise
from nise_2017_b200 import synth

pytestmark = pytest.mark.gpu

SPARSE_FP32 = 3e-6  # FP32 series vs the exact propagator


@pytest.mark.parametrize("n, cut", [(1, 2.0), (7, 2.0), (8, 2.0), (9, 2.0), (9, 1e6), (33, 60.0), (100, 2.0), (193, 2.0), (300, 2.0), (385, 2.0)])
def test_row_owner_on_small_lattices(n, cut, tmp_path):
    frames = 470
    files = synth.write(synth.c1_spec(n_sites=n, frames=frames, seed=n + 2), str(tmp_path))
    kw = synth.c1_keywords(Singles=n, Length=frames, Couplingcut=cut, RunTimes="9 0 0", Samplerate=1)
    out = {}
    for key, engine in ((0, {}), (15, {"kernel_config": 15}), (14, {"kernel_config": 14}), (13, {"kernel_config": 13}),
                        (64, {"precision": nise.FP64})):
        with nise.Context(nise.params_from_keywords(kw, files, **engine)) as c:
            c.load_files()
            re, im, _ = c.absorption()
            out[key] = re + 1j * im
    assert np.array_equal(out[0], out[15])
    for key in (13, 14, 15):
        assert helpers.rel(out[key], out[64]) < SPARSE_FP32
