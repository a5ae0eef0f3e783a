"""nise_propagate on either side of the number of vectors from which a thread per
vector is faster than a CTA: every vector's step is the same in a call of few
and of many, in FP32 bitwise."""
import numpy as np
import pytest

import helpers
import nise_2017_b200 as nise
from nise_2017_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prop, n, line", [("Coupling", 2, 5000), ("Coupling", 8, 20000), ("Sparse", 3, 7500), ("Sparse", 8, 20000),
                                           ("RK4", 2, 3400), ("RK4", 7, 11900), ("RK4", 8, 13600)])
def test_many_vectors(prop, n, line):
    rng = np.random.default_rng(n)
    h = rng.normal(0, 5, size=(line, n * (n + 1) // 2)).astype(np.float32)
    z = rng.normal(size=(2, line, n))
    for precision, dtype in ((nise.FP32, np.float32), (nise.FP64, np.float64)):
        x, y = z.astype(dtype)
        kw = synth.c0_keywords(Singles=n, Propagation=prop, Threshold=0)
        with nise.Context(nise.params_from_keywords(kw, precision=precision)) as c:
            few = [np.array(v) for v in c.propagate(h[:50], x[:50], y[:50])]
            for count in (line - 1, line):
                many = c.propagate(h[:count], x[:count], y[:count])
                for a, b in zip(few, many):
                    if precision == nise.FP32 and prop != "Sparse":
                        assert np.array_equal(a, b[:50])
                    else:
                        assert helpers.rel(b[:50], a) < (1e-6 if precision == nise.FP32 else 1e-13)
