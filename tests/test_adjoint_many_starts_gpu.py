"""The Trotter adjoint of few sites on either side of the number of start points from
which a thread per vector is faster than the scheduled kernels: the spectrum of
all start points is the sum of the halves', and the gradients of a spectrum that
is linear in the responses add up; the time grows less than the start points."""
import time

import numpy as np
import pytest

import helpers
import nise_2017_b200 as nise
from nise_2017_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 5, 8])
def test_many_start_points(n, tmp_path):
    few, most, T = 100, 3000, 16
    frames = 4 * most + T + 2
    files = synth.write(synth.c3_spec(n_sites=n, frames=frames, geometry=synth.CLUSTER, seed=n), str(tmp_path))
    shift = np.linspace(-3, 3, n)
    best, out = {}, {}
    for begin, end in ((0, few), (few, most), (0, most)):
        kw = synth.c3_keywords(Singles=n, Length=frames, RunTimes="%d 0 0" % T, Samplerate=4, BeginPoint=begin, EndPoint=end)
        with nise.Context(nise.params_from_keywords(kw, files)) as c:
            c.load_files()
            w, sr, si = c.absorption_model(shift, 1.05, 900.0)
            up = np.cos(np.arange(len(w)))
            times = []
            for _ in range(5):
                t = time.perf_counter()
                c.absorption_model(shift, 1.05, 900.0)
                g = c.backward_absorption(shift, 1.05, 900.0, up, -up)
                times.append(time.perf_counter() - t)
            best[begin, end] = min(times)
            # the spectrum is divided by the number of samples, the last start point's
            out[begin, end] = end * np.concatenate([sr, si, g[0], [g[1], g[2]]])
    assert helpers.rel(out[0, few] + out[few, most], out[0, most]) < 1e-10
    assert best[0, most] < 0.3 * most / few * best[0, few], best


@pytest.mark.parametrize("n, geometry", [(300, synth.LATTICE), (5, synth.CLUSTER)])
def test_next_to_no_steps(n, geometry, tmp_path):
    """RunTimes 1: no schedule is made for a job without steps (and 2 and 9 on either
    side of its line for 5 sites), the spectrum is that of the FP64 absorption."""
    files = synth.write(synth.c3_spec(n_sites=n, frames=60, geometry=geometry, seed=n), str(tmp_path))
    best = {}
    for T in (1, 2, 9, 16):
        kw = synth.c3_keywords(Singles=n, Length=60, RunTimes="%d 0 0" % T, Samplerate=3, EndPoint=14, FFT=64, Lifetime=900)
        with nise.Context(nise.params_from_keywords(kw, files, precision=nise.FP64)) as c:
            c.load_files()
            times = []
            for _ in range(5):
                t = time.perf_counter()
                w, sr, si = c.absorption_model(np.zeros(n), 1.0, 900.0)
                times.append(time.perf_counter() - t)
            best[T] = min(times)
            re, im, count = c.absorption()
            _, er, ei = c.absorption_fft(re, im, count)
        assert helpers.rel(sr + 1j * si, er + 1j * ei) < 1e-9
    if n == 300:
        assert best[1] < 0.6 * best[2], best
