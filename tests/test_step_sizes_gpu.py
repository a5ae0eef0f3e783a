"""nise_propagate on a CTA per vector, over the sizes where its split changes:
one site, one and several warps of rows or rotations, one vector and many, and
above the size whose coefficients fit shared memory (240 sites: a thread per
vector takes over for the Trotter scheme).  Against the oracle's per-vector step,
bitwise in FP32 for the schemes that reproduce the reference's operations.
"""
import numpy as np
import pytest

import helpers
import nise_2017_b200 as nise
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prop", ["Coupling", "RK4", "Sparse"])
@pytest.mark.parametrize("n, nvec", [(1, 3), (2, 1), (16, 3), (33, 5), (64, 2), (65, 2), (130, 2), (240, 1)])
def test_step_sizes(prop, n, nvec):
    rng = np.random.default_rng(n)
    kw = dict(Propagation=prop, Singles=n, Length=100, Samplerate=10, Timestep=2, RunTimes="10 0 0", Trotter=2,
              Couplingcut=1.0, Threshold=0, Technique="Absorption", MinFrequencies="-100 0 0", MaxFrequencies="100 0 0")
    iu = np.triu_indices(n)
    H = rng.normal(0, 2.0, size=(nvec, len(iu[0]))).astype(np.float32)
    H[:, iu[0] == iu[1]] *= 10
    # the propagators differ on purpose in what |J| <= Couplingcut does: cleared here, as the frame readers do
    H[:, iu[0] != iu[1]] *= np.abs(H[:, iu[0] != iu[1]]) > 1.0
    re = rng.normal(size=(nvec, n)).astype(np.float32)
    im = rng.normal(size=(nvec, n)).astype(np.float32)
    po = oracle.params(kw, {})
    for prec, dt, build in ((nise.FP32, np.float32, "f32"), (nise.FP64, np.float64, "f64")):
        with nise.Context(nise.params_from_keywords(kw, precision=prec)) as c:
            gr, gi = c.propagate(H, re.astype(dt), im.astype(dt), 1)
        orr, oii = re.astype(dt).copy(), im.astype(dt).copy()
        for v in range(nvec):
            a, b = orr[v].copy(), oii[v].copy()
            oracle.lib(build).oracle_propagate_vector(oracle.ctypes.byref(po), H[v].ctypes.data_as(
                oracle.ctypes.POINTER(oracle.ctypes.c_float)), a.ctypes.data, b.ctypes.data, 1)
            orr[v], oii[v] = a, b
        if prop == "Sparse":
            assert helpers.rel(gr + 1j * gi, orr + 1j * oii) < (2e-6 if prec == nise.FP32 else 1e-11)
        elif prec == nise.FP32:
            assert np.array_equal(gr, orr) and np.array_equal(gi, oii)
        else:
            assert helpers.rel(gr + 1j * gi, orr + 1j * oii) < 1e-12
