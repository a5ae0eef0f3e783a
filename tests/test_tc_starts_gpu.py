"""The tensor-core apply with all start points in step (a batched job whose
propagators are all held) against one start point at a time, frame by frame
(plain mode): the same column arithmetic, so bitwise the same vectors.

130 sites leave two rows in the second 128-row tile, 257 one in the third; one
start point, and more than fill a column group.
"""
import numpy as np
import pytest

import nise_2017_b200 as nise
from nise_2017_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, tmax, sample, end", [(130, 20, 7, 0), (130, 12, 11, 1), (257, 9, 12, 0)])
def test_starts_in_step_equal_plain(n, tmax, sample, end, tmp_path):
    files = synth.write(synth.c0_spec(n_sites=n, frames=90, geometry=synth.CLUSTER, spacing=6.0, seed=n + tmax), str(tmp_path))
    kw = synth.c0_keywords(Singles=n, Length=90, RunTimes="%d 0 0" % tmax, Samplerate=sample, Propagation="Sparse",
                           Threshold=0, EndPoint=end)
    out = []
    for mode in (nise.BATCHED, nise.PLAIN):
        with nise.Context(nise.params_from_keywords(kw, files, launch_mode=mode)) as c:
            c.load_files()
            re, im, count = c.absorption()
        out.append((np.stack([re, im]), count))
    assert out[0][1] == out[1][1] >= 1
    assert np.array_equal(out[0][0], out[1][0])
