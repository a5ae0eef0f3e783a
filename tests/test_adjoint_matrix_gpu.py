"""The Trotter adjoint around the sizes where its kernels change: matrices of a
window of four steps in shared memory up to a 258-site chain (rotations and phases
apart from 259 on), matrices of one step up to about 1700 couplings, rotations in
shared memory up to about 4600 and from global memory above.

Against the engine's FP64 absorption and central differences, as the scheduled
adjoint's test.
"""
import pytest

import test_adjoint_schedule_gpu as scheduled
from nise_2017_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, geometry, tmax", [(258, synth.CHAIN, 10), (259, synth.CHAIN, 10), (58, synth.CLUSTER, 6),
                                               (64, synth.CLUSTER, 6), (100, synth.CLUSTER, 6)])
def test_adjoint_kernels(n, geometry, tmax, tmp_path):
    cut = 0.1 if geometry == synth.CHAIN else 0.0
    scheduled.test_scheduled_adjoint(n, geometry, cut, tmax, tmp_path)
