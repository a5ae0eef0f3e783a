"""The Trotter adjoint on the scheduled rotations: windows of four time steps
(chains) and single steps (wide coupling lists), sites without any coupling, and
lengths that leave a remainder of the window and of the checkpoint interval.

The model equals the engine's FP64 absorption at zero shifts; the gradient
equals central differences of the model (one Richardson step) per component.
"""
import numpy as np
import pytest

import helpers
import nise_2017_b200 as nise
from nise_2017_b200 import synth

pytestmark = pytest.mark.gpu

MODEL = 1e-11     # the same scheme in FP64
GRADIENT = 1e-6   # of the largest component, as the other adjoint tests


@pytest.mark.parametrize("n, geometry, cut, tmax", [(1, synth.CHAIN, 0.1, 7), (2, synth.CHAIN, 0.1, 2),
                                                    (7, synth.CLUSTER, 6.0, 9), (33, synth.CLUSTER, 0.1, 38),
                                                    (40, synth.CHAIN, 0.1, 71), (41, synth.CHAIN, 0.1, 33)])
def test_scheduled_adjoint(n, geometry, cut, tmax, tmp_path):
    frames = tmax + 45
    files = synth.write(synth.c0_spec(n_sites=n, frames=frames, geometry=geometry, spacing=6.0, seed=80 + n + tmax),
                        str(tmp_path))
    kw = synth.c0_keywords(Singles=n, Length=frames, RunTimes="%d 0 0" % tmax, Samplerate=21, Couplingcut=cut, FFT=128)
    rng = np.random.default_rng(n)
    with nise.Context(nise.params_from_keywords(kw, files, precision=nise.FP64)) as c:
        c.load_files()
        re, im, count = c.absorption()
        w, sr, si = c.absorption_fft(re, im, count)
        mw, mr, mi = c.absorption_model(np.zeros(n), 1.0, float(kw["Lifetime"]))
        assert np.array_equal(w, mw)
        assert helpers.rel(mr + 1j * mi, sr + 1j * si) < MODEL
        shift, scale, life = rng.normal(0, 5, n), 1.1, 700.0
        gr, gi = rng.normal(size=len(w)), rng.normal(size=len(w))

        def loss(s, k):
            _, a, b = c.absorption_model(s, k, life)
            return float(a @ gr + b @ gi)

        g, gs, _ = c.backward_absorption(shift, scale, life, gr, gi)

        def slope(f, h):
            d = lambda e: (f(e) - f(-e)) / (2 * e)
            return (4 * d(h) - d(2 * h)) / 3

        sites = sorted({0, n // 2, n - 1})
        fd = []
        for a in sites:
            e = np.eye(n)[a]
            fd.append(slope(lambda x: loss(shift + x * e, scale), 0.05))
        top = max(np.abs(g).max(), abs(gs))
        assert np.abs(np.array(fd) - g[sites]).max() < GRADIENT * top
        assert abs(slope(lambda x: loss(shift, scale + x), 1e-3) - gs) < GRADIENT * max(top, 1.0)
