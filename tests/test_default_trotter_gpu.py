"""The default Trotter kernel of an absorption job against those that can be asked for
(a warp per vector, two vectors per warp, rows of 32 and 64 operations): the
same responses (in FP32 bitwise), and no more than a quarter slower than the fastest, where the
rule changes: the schedule of dense couplings in shared memory or too large for
it, one wave of CTAs or a short second one, static couplings on rows of 64.  (The
lines are drawn within 10 %; on the wrong side of them kernels are 1.4 to 3 times
slower.)"""
import numpy as np
import pytest

import helpers
import nise_2017_b200 as nise
from nise_2017_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, static, points, precision", [
    (100, False, 60, nise.FP32), (100, False, 150, nise.FP32), (100, False, 600, nise.FP32), (128, False, 2, nise.FP32),
    (80, False, 150, nise.FP64), (33, False, 600, nise.FP32), (64, False, 800, nise.FP32), (120, False, 2, nise.FP64),
    (100, True, 390, nise.FP32), (200, True, 150, nise.FP32), (200, True, 200, nise.FP32), (400, True, 200, nise.FP64),
    (400, True, 390, nise.FP64), (128, True, 450, nise.FP32)])
def test_default_is_near_the_fastest(n, static, points, precision, tmp_path):
    frames = 33 + 4 * points
    if static:
        spec, kw = synth.c1_spec(n_sites=n, frames=frames, seed=n), synth.c1_keywords()
    else:
        spec, kw = synth.c2_spec(n_sites=n, frames=frames, ham_type=synth.FULL, dipole_frames=0, seed=n), synth.c2_keywords()
    files = synth.write(spec, str(tmp_path))
    kw.update(Singles=n, Length=frames, RunTimes="24 0 0", Samplerate=4, EndPoint=points, Technique="Absorption",
              Propagation="Coupling", HamiltonianType="Coupling" if static else "Full")
    ms, out = {}, {}
    for config in (0, 32, 35) + ((34, 36) if static else ()):
        with nise.Context(nise.params_from_keywords(kw, files, precision=precision, kernel_config=config)) as c:
            c.load_files()
            ms[config] = min((c.absorption(), c.timing()[0])[1] for _ in range(6))
            out[config] = c.absorption()
        if precision == nise.FP32:
            assert np.array_equal(out[config][0], out[0][0]) and np.array_equal(out[config][1], out[0][1])
        else:  # the kernels contract products and sums in their own ways
            assert helpers.rel(out[config][0], out[0][0]) < 1e-12
    assert ms[0] <= 1.25 * min(ms.values()), ms
