"""Exact jobs with static couplings and fewer vectors than a wave of 8-vector CTAs:
the default's error against FP64 is that of the Taylor series on the 4-vector
kernel (kernel_config 12), on either side of the size where the row-owner kernel
takes over (300 sites), with all vectors on 1-vector CTAs and with some on 8.  The
bound is 1.5 times: the same terms, rounded in another order (the Chebyshev
recurrence is 4 times worse)."""
import pytest

import helpers
import nise_2017_b200 as nise
from nise_2017_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, points", [(299, 60), (300, 60), (420, 30), (600, 95), (1024, 60)])
def test_few_vectors_keep_the_taylor_rounding(n, points, tmp_path):
    frames = 129 + 10 * (points - 1)
    files = synth.write(synth.c1_spec(n_sites=n, frames=frames, seed=n), str(tmp_path))
    kw = synth.c1_keywords(Singles=n, Length=frames, RunTimes="128 0 0", Samplerate=10)
    out = {}
    for key, engine in ((0, {}), (12, {"kernel_config": 12}), (64, {"precision": nise.FP64})):
        with nise.Context(nise.params_from_keywords(kw, files, **engine)) as c:
            c.load_files()
            re, im, _ = c.absorption()
            out[key] = re + 1j * im
    assert helpers.rel(out[0], out[64]) <= 1.5 * helpers.rel(out[12], out[64])
