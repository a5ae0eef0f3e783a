"""The coupling pattern of a Full trajectory is found whichever frame it is in.

A coupling above Couplingcut in one frame only belongs to the pattern (the
reference tests |J| > Couplingcut frame by frame, propagate.c:853).  One frame
of each trajectory carries one strong coupling; if the scan missed it, the
Trotter responses would miss its rotation and differ from the oracle's by far
more than the summation order.
"""
import numpy as np
import pytest

import helpers
import nise_2017_b200 as nise
import oracle
from nise_2017_b200 import synth

pytestmark = pytest.mark.gpu

SUM_ORDER = 1e-11  # same float operations, FP64 sums in another order


@pytest.mark.parametrize("n, frames, hot", [(2, 33, 0), (3, 40, 31), (23, 70, 68), (23, 70, 7), (24, 600, 333)])
def test_one_strong_coupling_in_one_frame(n, frames, hot, tmp_path):
    files = synth.write(synth.c0_spec(n_sites=n, frames=frames, j_nn=0.0, j_sigma=0.0, seed=n + frames), str(tmp_path))
    rec = np.fromfile(files["energy"], np.float32).reshape(frames, -1)
    a, b = 0, n - 1
    rec[hot, 1 + b + a * (2 * n - a - 1) // 2] = -40.0
    rec.tofile(files["energy"])
    kw = synth.c0_keywords(Singles=n, Length=frames, RunTimes="16 0 0", Samplerate=1)
    with nise.Context(nise.params_from_keywords(kw, files)) as c:
        c.load_files()
        re, im, count = c.absorption()
    ore, oim, ocount = oracle.absorption(oracle.params(kw, files), "f32a64")
    assert count == ocount
    assert helpers.rel(re + 1j * im, ore + 1j * oim) < SUM_ORDER
