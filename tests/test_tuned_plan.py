"""A plan and the autotuner's table, which all contexts of a process share.

Another context's tuner may enter a configuration while a plan is being made, so
the plan reads the table before it builds any layout and not again; and a
configuration tuned for the same number of sites need not fit this job's
couplings."""
import os
import re

import numpy as np
import pytest

import helpers
import nise_2017_b200 as nise
from nise_2017_b200 import synth

SOURCE = os.path.join(os.path.dirname(os.path.abspath(nise.__file__)), "csrc", "absrun.cpp")


def test_the_table_is_read_before_the_layouts():
    plan = open(SOURCE).read().split("int AbsRun::plan(")[1].split("\n}\n")[0]
    reads = [m.start() for m in re.finditer(r"g_tuned|\btuned\(|read_tuned\(", plan)]
    branches = [m.start() for m in re.finditer(r"scheme = SCHEME_", plan)]
    # at most one read in each scheme's branch, none after the last branch
    assert reads and max(reads) < plan.index("config = default_config(")
    for a, b in zip(branches, branches[1:] + [len(plan)]):
        assert sum(a < r < b for r in reads) <= 1


@pytest.mark.gpu
def test_tuned_for_fewer_couplings(tmp_path):
    """300 sites with 11 neighbours tuned (the row-owner kernel is the fastest), then
    300 sites with 100, whose tables do not fit that kernel."""
    n, frames = 300, 40
    files = synth.write(synth.c1_spec(n_sites=n, frames=frames, jcut=0.0, seed=5), str(tmp_path))
    out = {}
    for cut in (2.0, 0.12):
        kw = synth.c1_keywords(Singles=n, Length=frames, Couplingcut=cut, RunTimes="8 0 0", Samplerate=1)
        for precision in (nise.FP32, nise.FP64):
            with nise.Context(nise.params_from_keywords(kw, files, precision=precision)) as c:
                c.load_files()
                if precision == nise.FP32 and cut == 2.0:
                    c.tune()
                re_, im, _ = c.absorption()
                out[precision] = re_ + 1j * im
        assert np.abs(out[nise.FP64]).max() > 0
        assert helpers.rel(out[nise.FP32], out[nise.FP64]) < 3e-6
