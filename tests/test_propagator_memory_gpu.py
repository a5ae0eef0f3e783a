"""What a per-frame exact job keeps on the device, next to those of other jobs of a
batch: the frames' propagators, and a workspace no larger than the eigenvectors
and QR workspace that it replaced (148 frames of 16 N^2 bytes, or 1 GB).  A call by
itself may use more while it runs, with the same result."""
import numpy as np
import pytest
import torch

import nise_2017_b200 as nise
from nise_2017_b200 import synth

pytestmark = pytest.mark.gpu


def test_workspace_of_a_held_job(tmp_path):
    n, frames = 700, 330
    files = synth.write(synth.c2_spec(n_sites=n, frames=frames, ham_type=synth.FULL, dipole_frames=0, seed=9), str(tmp_path))
    kw = synth.c2_keywords(Singles=n, Length=frames, RunTimes="20 0 0", Samplerate=100, Technique="Absorption",
                           HamiltonianType="Full", Propagation="Sparse", Threshold=0)
    with nise.Context(nise.params_from_keywords(kw, files)) as c:
        c.load_files()
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        with nise.Batch([c]) as b:
            held = before - torch.cuda.mem_get_info()[0]
            b.run()
            batch = b.result(0)
        alone = c.absorption()
    propagators = 8 * n * n * frames
    assert held < propagators + max(1 << 30, 148 * 16 * n * n) + (1 << 29)
    assert np.array_equal(batch[0], alone[0]) and np.array_equal(batch[1], alone[1])
