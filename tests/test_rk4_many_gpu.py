"""RK4 absorption on either side of the number of start points from which a thread per
vector is faster than a thread per site row: in FP32 the response of all start
points is the sum of the halves' (the order of the sum alone differs), and the
time grows less than the start points."""
import numpy as np
import pytest

import helpers
import nise_2017_b200 as nise
from nise_2017_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3])
@pytest.mark.parametrize("precision", [nise.FP32, nise.FP64])
def test_many_start_points(n, precision, tmp_path):
    most, few, T = 4000, 400, 32
    frames = 3 * most + T
    files = synth.write(synth.c2_spec(n_sites=n, frames=frames, ham_type=synth.FULL, dipole_frames=0, seed=n), str(tmp_path))
    ms, out = {}, {}
    for begin, end in ((0, few), (few, most), (0, most)):
        kw = synth.c2_keywords(Singles=n, Length=frames, Technique="Absorption", HamiltonianType="Full", Propagation="RK4",
                               RunTimes="%d 0 0" % T, Samplerate=3, BeginPoint=begin, EndPoint=end)
        with nise.Context(nise.params_from_keywords(kw, files, precision=precision)) as c:
            c.load_files()
            ms[begin, end] = min((c.absorption(), c.timing()[0])[1] for _ in range(5))
            re, im, _ = c.absorption()
            out[begin, end] = re + 1j * im
    assert helpers.rel(out[0, few] + out[few, most], out[0, most]) < 1e-12
    assert ms[0, most] < 0.35 * most / few * ms[0, few], ms
