"""The exact propagators of per-frame Hamiltonians (propagate_vec_DIA,
propagate.c:60-125) from Taylor polynomials and doublings.

Sizes below, at and above the kernel's tile (64 sites) and thread block (4
sites); time steps that take the short polynomial, the long one and several
doublings (||H|| f about 0.05, 0.5 and 6).  FP64 against numpy
eigendecompositions, and against the engine's own eigenvectors
(kernel_config 2).
"""
import pytest

import helpers
import nise_2017_b200 as nise
import oracle
from nise_2017_b200 import synth

pytestmark = pytest.mark.gpu

EXACT = 1e-9  # the eigen route's bound against the FP64 restatement


def absorb(kw, files, **engine):
    with nise.Context(nise.params_from_keywords(kw, files, precision=nise.FP64, **engine)) as c:
        c.load_files()
        re, im, n = c.absorption()
    return re + 1j * im, n


@pytest.mark.parametrize("n, dt", [(1, 2), (2, 100), (4, 2), (5, 20), (36, 1), (63, 2), (64, 20), (65, 2), (65, 200),
                                   (121, 2), (130, 20)])
def test_propagators_match_eigenvectors(n, dt, tmp_path):
    files = synth.write(synth.c0_spec(n_sites=n, frames=40, dt_fs=dt, geometry=synth.CLUSTER, spacing=6.0, seed=90 + n + dt),
                        str(tmp_path))
    kw = synth.c0_keywords(Singles=n, Length=40, Timestep=dt, RunTimes="9 0 0", Samplerate=12, Propagation="Sparse",
                           Threshold=0)
    ours, count = absorb(kw, files)
    eig, _ = absorb(kw, files, kernel_config=2)
    ex_re, ex_im, ex_count = oracle.absorption_exact(kw, files)
    assert count == ex_count
    assert helpers.rel(ours, ex_re + 1j * ex_im) < EXACT
    assert helpers.rel(ours, eig) < EXACT
