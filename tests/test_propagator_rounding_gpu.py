"""The propagators of per-frame Hamiltonians where the step is many doublings
long: two sites 1500 cm^-1 away from the others and from each other, Timestep 200
and 2000 fs (7 and 10 doublings).  An eigenvalue's own rounding is eps ||H|| f, and
the bound is four times that: the doublings must not add to it."""
import numpy as np
import pytest

import helpers
import nise_2017_b200 as nise
import oracle
from nise_2017_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, dt", [(40, 200), (65, 200), (40, 2000), (65, 2000)])
def test_doublings_keep_the_rounding(n, dt, tmp_path):
    files = synth.write(synth.c0_spec(n_sites=n, frames=40, dt_fs=2.0, geometry=synth.CLUSTER, spacing=6.0, seed=40 + n),
                        str(tmp_path))
    rec = np.fromfile(files["energy"], np.float32).reshape(40, -1)
    diagonal = [1 + a * n - a * (a - 1) // 2 for a in range(n)]
    rec[:, diagonal[3]] += 1500
    rec[:, diagonal[7]] -= 1500
    rec.tofile(files["energy"])
    kw = synth.c0_keywords(Singles=n, Length=40, Timestep=dt, RunTimes="9 0 0", Samplerate=12, Propagation="Sparse",
                           Threshold=0)
    with nise.Context(nise.params_from_keywords(kw, files, precision=nise.FP64)) as c:
        c.load_files()
        re, im, _ = c.absorption()
    ex_re, ex_im, _ = oracle.absorption_exact(kw, files)
    bound = 4 * np.finfo(np.float64).eps * 1500 * 2 * np.pi * 2.99792458e-5 * dt
    assert helpers.rel(re + 1j * im, ex_re + 1j * ex_im) < bound
