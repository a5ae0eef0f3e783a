"""Exact propagation with very many static couplings: 46 to 106 neighbours a row
at 300 to 512 sites.  The row-owner kernel's tables (three slots in 16 bytes)
still fit shared memory there; those of the 8-vector sliced-ELL kernel (8 bytes a
slot) do not, and at 100 and more neighbours neither do those of the 1-vector
kernel that takes a job's last vectors.  Few vectors, between one vector and
eight per SM, and whole waves.  FP32 against the FP64 context."""
import numpy as np
import pytest

import helpers
import nise_2017_b200 as nise
from nise_2017_b200 import synth

pytestmark = pytest.mark.gpu

SPARSE_FP32 = 3e-6  # FP32 series vs the exact propagator


@pytest.mark.parametrize("n, cut, points", [(300, 0.15, 12), (400, 0.25, 100), (512, 0.4, 12), (400, 0.25, 400),
                                            (300, 0.12, 12), (300, 0.12, 100), (300, 0.12, 400)])
def test_dense_static_couplings(n, cut, points, tmp_path):
    frames = points + 9
    files = synth.write(synth.c1_spec(n_sites=n, frames=frames, jcut=0.0, seed=5), str(tmp_path))
    kw = synth.c1_keywords(Singles=n, Length=frames, Couplingcut=cut, RunTimes="8 0 0", Samplerate=1)
    out = []
    for precision in (nise.FP32, nise.FP64):
        with nise.Context(nise.params_from_keywords(kw, files, precision=precision)) as c:
            c.load_files()
            re, im, count = c.absorption()
            assert count == points + 1
            out.append(re + 1j * im)
    assert np.abs(out[1]).max() > 0
    assert helpers.rel(out[0], out[1]) < SPARSE_FP32
