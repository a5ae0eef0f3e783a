"""Trotter steps scheduled as rows of independent operations, a warp per vector:
the reference's float operations in its order on every site (propagate.c:821-899),
so FP32 results equal the oracle's up to the order of the FP64 sums.

No coupling at all, one, chains (few operations per row), dense couplings (full
rows, more than one warp's worth of sites), static and per-frame coefficients.
"""
import pytest

import helpers
import nise_2017_b200 as nise
import oracle
from nise_2017_b200 import synth

pytestmark = pytest.mark.gpu

SUM_ORDER = 1e-10  # same float operations, FP64 sums in another order
FP64 = 1e-11       # the same formulas in FP64


def trajectory(tmp_path, n, geometry, ham, frames, seed):
    static = ham == "Coupling"
    return synth.write(synth.c0_spec(n_sites=n, frames=frames, geometry=geometry, spacing=6.0, seed=seed,
                                     ham_type=synth.COUPLING if static else synth.FULL, dipole_frames=1 if static else 0,
                                     mu_jitter=0.0 if static else 0.05), str(tmp_path))


SYSTEMS = [(1, synth.CHAIN, "Full", 0.1), (2, synth.CHAIN, "Full", 0.1), (9, synth.CLUSTER, "Coupling", 1e6),
           (16, synth.CHAIN, "Full", 0.1), (33, synth.CLUSTER, "Full", 0.1), (40, synth.CLUSTER, "Coupling", 0.1),
           (70, synth.CLUSTER, "Coupling", 0.1)]


@pytest.mark.parametrize("n, geometry, ham, cut", SYSTEMS[1:])
def test_2d_singles(n, geometry, ham, cut, tmp_path):
    files = trajectory(tmp_path, n, geometry, ham, 60, 600 + n)
    kw = synth.c2_keywords(Singles=n, Length=60, RunTimes="5 0 5", Samplerate=23, HamiltonianType=ham, Couplingcut=cut,
                           Technique="noEAIR", Trotter=3)
    for precision, build, tol in ((nise.FP32, "f32a64", SUM_ORDER), (nise.FP64, "f64", FP64)):
        with nise.Context(nise.params_from_keywords(kw, files, precision=precision)) as c:
            c.load_files()
            response, count = c.twodir()
        want, wcount = oracle.twodir(oracle.params(kw, files), build)
        assert count == wcount
        assert helpers.rel2d(response, want) < tol


@pytest.mark.parametrize("n, geometry, ham, cut", SYSTEMS)
def test_absorption_default_and_forced(n, geometry, ham, cut, tmp_path):
    """The default configuration, rows of 32 and rows of 64 (35, 36) against the thread per vector (1)."""
    files = trajectory(tmp_path, n, geometry, ham, 60, 700 + n)
    kw = synth.c0_keywords(Singles=n, Length=60, RunTimes="9 0 0", Samplerate=13, HamiltonianType=ham, Couplingcut=cut)
    for precision, build in ((nise.FP32, "f32a64"), (nise.FP64, "f64")):
        got = {}
        for config in (0, 1, 35, 36):
            with nise.Context(nise.params_from_keywords(kw, files, precision=precision, kernel_config=config)) as c:
                c.load_files()
                re, im, count = c.absorption()
            got[config] = re + 1j * im
        ore, oim, ocount = oracle.absorption(oracle.params(kw, files), build)
        assert count == ocount
        assert helpers.rel(got[1], ore + 1j * oim) < 1e-11
        for config in (0, 35, 36):
            if precision == nise.FP32:
                assert (got[config] == got[1]).all()
            else:
                assert helpers.rel(got[config], got[1]) < FP64


@pytest.mark.parametrize("tech", ["LD", "DOS", "CD"])
@pytest.mark.parametrize("n, geometry, ham, cut", [SYSTEMS[1], SYSTEMS[3], SYSTEMS[4], SYSTEMS[5]])
def test_linear_techniques(tech, n, geometry, ham, cut, tmp_path):
    files = trajectory(tmp_path, n, geometry, ham, 40, 800 + n)
    files.update(synth.write_positions(str(tmp_path), n, 40, seed=n))
    kw = synth.c0_keywords(Singles=n, Length=40, RunTimes="7 0 0", Samplerate=15, HamiltonianType=ham, Couplingcut=cut,
                           Technique=tech)
    for precision, build in ((nise.FP32, "f32a64"), (nise.FP64, "f64")):
        with nise.Context(nise.params_from_keywords(kw, files, precision=precision)) as c:
            c.load_files()
            re, im, count = c.linear()
        want = oracle.linear(oracle.params(kw, files), build)
        assert count == want[2]
        assert helpers.rel(re + 1j * im, want[0] + 1j * want[1]) < SUM_ORDER
