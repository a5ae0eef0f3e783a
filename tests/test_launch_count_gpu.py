"""The kernels that a per-frame exact job counts (nise_last_timing)."""
import pytest

import nise_2017_b200 as nise
from nise_2017_b200 import synth

pytestmark = pytest.mark.gpu


def test_exact_job_counts_its_kernels(tmp_path):
    """The propagators (by eigenvectors: the eigensolver and the build of U), the
    apply and the response sum."""
    files = synth.write(synth.c0_spec(n_sites=12, frames=200, geometry=synth.CLUSTER, seed=9), str(tmp_path))
    kw = synth.c0_keywords(Singles=12, Length=200, RunTimes="20 0 0", Samplerate=10, Propagation="Sparse", Threshold=0)
    counts = {}
    for config in (0, 2):
        with nise.Context(nise.params_from_keywords(kw, files, kernel_config=config)) as c:
            c.load_files()
            c.absorption()
            counts[config] = c.timing()[2]
    assert counts == {0: 3, 2: 4}
