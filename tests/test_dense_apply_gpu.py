"""The dense one-step propagators applied per start point (absorption) and to all
vectors of a start point at once (linear techniques).

Absorption: one site; sizes about where two propagators no longer fit shared
memory (84 sites in FP64, 119 in FP32), where a thread takes all three vectors
(310 sites) and where the response warps share the rows' (930 sites).  CD, LD and DOS: fewer vectors than a column block,
a remainder of it, and several blocks per start point.
"""
import numpy as np
import pytest

import helpers
import nise_2017_b200 as nise
import oracle
from nise_2017_b200 import synth

pytestmark = pytest.mark.gpu

EXACT = 1e-9        # FP64 against the FP64 restatement, as the other eigen-route tests
SPARSE_FP32 = 3e-6  # FP32 vectors through exact propagators


@pytest.mark.parametrize("n, tmax", [(1, 5), (2, 1), (3, 9), (33, 12), (84, 6), (85, 6), (119, 5), (310, 3), (930, 3)])
def test_absorption_sizes(n, tmax, tmp_path):
    files = synth.write(synth.c0_spec(n_sites=n, frames=tmax + 16, geometry=synth.CHAIN, seed=n + tmax), str(tmp_path))
    kw = synth.c0_keywords(Singles=n, Length=tmax + 16, RunTimes="%d 0 0" % tmax, Samplerate=7, Propagation="Sparse",
                           Threshold=0)
    ex_re, ex_im, ex_count = oracle.absorption_exact(kw, files)
    for precision, config, tol in ((nise.FP64, 0, EXACT), (nise.FP32, 16, SPARSE_FP32)):
        with nise.Context(nise.params_from_keywords(kw, files, precision=precision, kernel_config=config)) as c:
            c.load_files()
            re, im, count = c.absorption()
        assert count == ex_count
        assert helpers.rel(re + 1j * im, ex_re + 1j * ex_im) < tol


@pytest.mark.parametrize("tech, n, points", [("LD", 2, 1), ("LD", 37, 9), ("DOS", 5, 3), ("DOS", 43, 6), ("CD", 7, 2),
                                             ("CD", 21, 8)])
def test_linear_sizes(tech, n, points, tmp_path):
    frames = 12 + 5 * points
    files = synth.write(synth.c0_spec(n_sites=n, frames=frames, geometry=synth.CLUSTER, spacing=6.0, seed=n), str(tmp_path))
    files.update(synth.write_positions(str(tmp_path), n, frames, seed=n))
    kw = synth.c0_keywords(Singles=n, Length=frames, RunTimes="8 0 0", Samplerate=5, EndPoint=points, Propagation="Sparse",
                           Threshold=0, Technique=tech)
    p = oracle.params(kw, files)
    o64 = oracle.linear(p, "f64")
    o32 = oracle.linear(p, "f32a64")
    want = np.asarray(o64[0]) + 1j * np.asarray(o64[1])
    own = helpers.rel(np.asarray(o32[0]) + 1j * np.asarray(o32[1]), want)
    for precision, tol in ((nise.FP64, EXACT), (nise.FP32, max(1.5 * own, 1e-5))):
        with nise.Context(nise.params_from_keywords(kw, files, precision=precision)) as c:
            c.load_files()
            re, im, count = c.linear()
        assert count == points
        assert helpers.rel(re + 1j * im, want) < tol
