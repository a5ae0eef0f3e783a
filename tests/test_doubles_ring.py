"""The ring of coupling records of the two-vector doubles kernel
(k2d_doubles_pair, csrc/twodir.cu).

A warp keeps 64 records in shared memory.  Before the couplings k .. k + 31 it
writes the records k + 32 .. k + 63 over those of k - 32 .. k - 1, each lane one
of them, and every lane reads the records of the couplings it applies.  The
warp that owns a segment synchronises after every coupling, the other one
(pair_free) not at all, so a lane that is ahead may write a record that another
one has still to read unless the warp synchronises before it writes.

On the CPU: every read of a slot and the write that replaces it must have a
synchronisation between them, with the statements of the kernel's source.  On
the GPU: the responses equal those of one vector at a time bitwise, at sizes
whose unsynchronised runs cross the chunks of 32 most often.
"""
import os
import re

import numpy as np
import pytest

import nise_2017_b200 as nise
from nise_2017_b200 import synth
from test_doubles_schedule import segments

SOURCE = os.path.join(os.path.dirname(os.path.abspath(nise.__file__)), "csrc", "twodir.cu")


def refill_statements():
    """The statements of the branch that refills the ring, in order."""
    body = re.search(r"if \(\(k & 31\) == 0\) \{(.*?)\n\s*\}\n", open(SOURCE).read(), re.S).group(1)
    body = re.sub(r"//[^\n]*", "", body)
    return [re.match(r"\s*(\w+)", x).group(1) for x in body.split(";") if x.strip()]


def unordered(pairs, half, statements):
    """Reads of a record that nothing orders before the write that replaces it."""
    epoch, read, bad = 0, {}, 0

    def sync():
        nonlocal epoch
        epoch += 1

    for a, k, end, owner in segments(pairs):
        sync()  # the barrier of the two warps
        while k < end:
            if k % 32 == 0:
                for st in statements:
                    if st == "__syncwarp":
                        sync()
                    elif st == "put":
                        bad += sum(read.pop((k + 32 + i) % 64, -1) == epoch for i in range(32))
            stop = min(end, (k | 31) + 1)
            for q in range(k, stop):
                read[q % 64] = epoch
                if half == owner:
                    sync()
            k = stop
    return bad


@pytest.mark.parametrize("n", [33, 48, 64])
def test_records_are_read_before_they_are_replaced(n):
    pairs = [(a, b) for a in range(n) for b in range(a + 1, n)]
    assert unordered(pairs, 1, ["put", "get", "__syncwarp"]) > 0  # a missing synchronisation is seen
    for half in (0, 1):
        assert unordered(pairs, half, refill_statements()) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("n", [48, 64])
def test_ring_refills_inside_unsynchronised_runs(n, tmp_path):
    s = synth.c2_spec(n_sites=n, frames=40, seed=700 + n)
    files = synth.write(s, str(tmp_path))
    kw = synth.c2_keywords(Singles=n, Length=40, RunTimes="6 0 6", Samplerate=13, Couplingcut=0.0, Trotter=3)
    out = []
    for config in (0, 0, 1):
        with nise.Context(nise.params_from_keywords(kw, files, kernel_config=config)) as c:
            c.load_files()
            out.append(c.twodir()[0])
    assert np.array_equal(out[0], out[2]) and np.array_equal(out[1], out[2])
