"""Two doubles vectors per warp (FP32, up to 64 sites) against one
(kernel_config 1): the same float operations in the same order, so the
responses are bitwise equal.

One column per lane up to 32 sites, two warps above; odd vector counts (the last
warp half empty: 9 + 9 tmax1), few couplings (pivots without any, runs shorter
than a step's look-ahead), more than the staged 64, and per-frame couplings.
"""
import numpy as np
import pytest

import nise_2017_b200 as nise
from nise_2017_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, tech, ham, cut", [(2, "2DIR", "Coupling", 0.1), (3, "2DUVvis", "Full", 0.1),
                                               (17, "2DIR", "Full", 0.1), (17, "2DIR", "Coupling", 12.0),
                                               (31, "2DUVvis", "Coupling", 0.1), (32, "2DIR", "Coupling", 0.1),
                                               (33, "2DIR", "Full", 4.0), (34, "2DUVvis", "Coupling", 0.1),
                                               (63, "2DIR", "Coupling", 2.0)])
def test_pairs_equal_single_vectors(n, tech, ham, cut, tmp_path):
    static = ham == "Coupling"
    s = synth.c2_spec(n_sites=n, frames=60, seed=500 + n, ham_type=synth.COUPLING if static else synth.FULL,
                      dipole_frames=1 if static else 0, mu_jitter=0.0 if static else 0.05)
    files = synth.write(s, str(tmp_path))
    kw = synth.c2_keywords(Singles=n, Length=60, RunTimes="4 0 4", Samplerate=25, Technique=tech, HamiltonianType=ham,
                           Couplingcut=cut, Trotter=2)
    out = []
    for config in (0, 1):
        with nise.Context(nise.params_from_keywords(kw, files, kernel_config=config)) as c:
            c.load_files()
            out.append(c.twodir()[0])
    assert np.abs(out[0]).max() > 0
    assert np.array_equal(out[0], out[1])
