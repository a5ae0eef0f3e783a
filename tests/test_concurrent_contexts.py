"""Contexts of different sizes on several threads at once.  A kernel's limit on
dynamic shared memory belongs to the process: set to one launch's size, it can be
lowered by another thread between that call and the launch, which then fails
("invalid argument", once in some ten thousand calls).  So there is one place that
sets it, to the same value always; and steps of several sizes run side by side."""
import glob
import os
import threading

import numpy as np
import pytest

import nise_2017_b200 as nise
from nise_2017_b200 import synth

CSRC = os.path.join(os.path.dirname(os.path.abspath(nise.__file__)), "csrc")


def test_one_place_sets_the_limit():
    calls = {os.path.basename(f): open(f).read().count("MaxDynamicSharedMemorySize") for f in glob.glob(CSRC + "/*")}
    assert {f: n for f, n in calls.items() if n} == {"common.cuh": 1}


@pytest.mark.gpu
@pytest.mark.parametrize("prop, sizes", [("Coupling", (16, 112, 150, 180, 200)), ("Sparse", (16, 160, 200, 250, 300)),
                                         ("RK4", (16, 160, 200, 250, 300))])
def test_steps_of_different_sizes(prop, sizes):
    rng = np.random.default_rng(3)
    work = []
    for n in sizes:
        h = rng.normal(0, 3.0, size=(1, n * (n + 1) // 2)).astype(np.float32)
        z = rng.normal(size=(2, 1, n)).astype(np.float32)
        c = nise.Context(nise.params_from_keywords(synth.c0_keywords(Singles=n, Propagation=prop, Threshold=0, Trotter=1)))
        work.append((c, h, z, c.propagate(h, z[0], z[1])))
    errors = []

    def run(c, h, z, ref):
        try:
            for _ in range(1500):
                got = c.propagate(h, z[0], z[1])
                assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=run, args=w) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for w in work:
        w[0].close()
    assert not errors, errors[0]
