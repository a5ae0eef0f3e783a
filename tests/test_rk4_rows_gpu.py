"""RK4 absorption with a thread per site row: the reference's operations in the
reference's order (propagate.c:311-366), so FP32 responses equal the oracle's up
to the order of the FP64 sums.

Sizes: one warp per vector up to 32 sites, several above; dense rows in shared
memory (33, 64 sites) and above it (200 sites); sparse rows of unequal length
(chains); 321 sites, one above what the row kernel takes.
"""
import pytest

import helpers
import nise_2017_b200 as nise
import oracle
from nise_2017_b200 import synth

pytestmark = pytest.mark.gpu

SUM_ORDER = 1e-11  # same float operations, FP64 sums in another order
FP64 = 1e-11       # the same formulas in FP64


@pytest.mark.parametrize("n, geometry, ham", [(2, synth.CHAIN, "Full"), (9, synth.CLUSTER, "Coupling"), (31, synth.CHAIN, "Full"),
                                              (32, synth.CLUSTER, "Full"), (33, synth.CLUSTER, "Full"),
                                              (64, synth.CLUSTER, "Full"), (200, synth.CLUSTER, "Full"),
                                              (320, synth.CHAIN, "Full"), (321, synth.CHAIN, "Full")])
def test_rows_match_oracle(n, geometry, ham, tmp_path):
    static = ham == "Coupling"
    s = synth.c0_spec(n_sites=n, frames=40, geometry=geometry, spacing=6.0, seed=70 + n,
                      ham_type=synth.COUPLING if static else synth.FULL, dipole_frames=1 if static else 0,
                      mu_jitter=0.0 if static else 0.05)
    files = synth.write(s, str(tmp_path))
    kw = synth.c0_keywords(Singles=n, Length=40, RunTimes="6 0 0", Samplerate=15, Propagation="RK4", Trotter=2,
                           HamiltonianType=ham)
    for precision, build, tol in ((nise.FP32, "f32a64", SUM_ORDER), (nise.FP64, "f64", FP64)):
        with nise.Context(nise.params_from_keywords(kw, files, precision=precision)) as c:
            c.load_files()
            re, im, count = c.absorption()
        ore, oim, ocount = oracle.absorption(oracle.params(kw, files), build)
        assert count == ocount
        assert helpers.rel(re + 1j * im, ore + 1j * oim) < tol
