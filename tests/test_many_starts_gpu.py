"""2D spectra of few sites with so many start points that a thread per vector fills
the GPU: the singles leave the rows of operations there.  The same responses in
FP32 (the sum of one call over the start points, of the halves of the range), and
the time grows less than the start points (rows: in proportion)."""
import numpy as np
import pytest

import helpers
import nise_2017_b200 as nise
from nise_2017_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tech, n, ham, precision", [("SEIR", 3, "Coupling", nise.FP32), ("SEIR", 5, "Full", nise.FP64),
                                                     ("GBIR", 8, "Coupling", nise.FP64), ("SEIR", 30, "Coupling", nise.FP32)])
def test_many_start_points(tech, n, ham, precision, tmp_path):
    most, few, T = 1500, 100, 16
    frames = 2 * T + 4 * most
    static = ham == "Coupling"
    files = synth.write(synth.c2_spec(n_sites=n, frames=frames, ham_type=synth.COUPLING if static else synth.FULL,
                                      dipole_frames=1 if static else 0, seed=n), str(tmp_path))
    ms, out = {}, {}
    for points in (few, most):
        kw = synth.c2_keywords(Singles=n, Length=frames, Technique=tech, HamiltonianType=ham, RunTimes="%d 0 %d" % (T, T),
                               Samplerate=4, EndPoint=points)
        with nise.Context(nise.params_from_keywords(kw, files, precision=precision)) as c:
            c.load_files()
            ms[points] = min((c.twodir(), c.timing()[0])[1] for _ in range(5))
            out[points] = c.twodir()[0]
    kw.update(BeginPoint=few)
    with nise.Context(nise.params_from_keywords(kw, files, precision=precision)) as c:
        c.load_files()
        rest = c.twodir()[0]
    assert helpers.rel2d(out[few] + rest, out[most]) < 1e-12  # the order of the sums over start points alone
    assert ms[most] < 0.5 * most / few * ms[few], ms
