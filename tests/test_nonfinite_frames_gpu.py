"""A frame with a NaN or an infinity above 120 sites ends in NISE_ERR_DEVICE (it
ran out of QR steps when every frame was diagonalised), in the absorption and in
the techniques that share nise_singles_tables; the context works on afterwards.
Up to 120 sites it is passed on to the result, as it always was.  Large finite
frames are no error."""
import numpy as np
import pytest

import nise_2017_b200 as nise
from nise_2017_b200 import synth

pytestmark = pytest.mark.gpu


def files_with(tmp_path, n, value, entry):
    files = synth.write(synth.c0_spec(n_sites=n, frames=40, geometry=synth.CLUSTER, spacing=6.0, seed=3), str(tmp_path))
    rec = np.fromfile(files["energy"], np.float32).reshape(40, -1)
    good = rec.copy()
    rec[5, entry] = value
    rec.tofile(files["energy"])
    return files, good


@pytest.mark.parametrize("precision", [nise.FP32, nise.FP64])
@pytest.mark.parametrize("technique", ["Absorption", "LD"])
@pytest.mark.parametrize("value, entry", [(np.nan, 1), (np.nan, 2), (np.inf, 3), (-np.inf, 1)])
def test_frames_that_are_not_finite(value, entry, technique, precision, tmp_path):
    n = 121
    files, good = files_with(tmp_path, n, value, entry)
    kw = synth.c0_keywords(Singles=n, Length=40, RunTimes="9 0 0", Samplerate=12, Propagation="Sparse", Threshold=0,
                           Technique=technique)
    with nise.Context(nise.params_from_keywords(kw, files, precision=precision)) as c:
        call = c.absorption if technique == "Absorption" else c.linear
        c.load_files()
        with pytest.raises(nise.NiseError) as e:
            call()
        assert e.value.code == -4  # NISE_ERR_DEVICE
        c.set_trajectory(good.view(np.uint8), np.fromfile(files["dipole"], np.uint8))
        assert np.all(np.isfinite(call()[0]))


def test_small_and_large_finite(tmp_path):
    kw = synth.c0_keywords(Singles=24, Length=40, RunTimes="9 0 0", Samplerate=12, Propagation="Sparse", Threshold=0)
    files, _ = files_with(tmp_path, 24, np.nan, 1)
    with nise.Context(nise.params_from_keywords(kw, files)) as c:
        c.load_files()
        assert not np.all(np.isfinite(c.absorption()[0]))
    files, _ = files_with(tmp_path, 130, 1e7, 1)
    kw["Singles"] = 130
    with nise.Context(nise.params_from_keywords(kw, files, precision=nise.FP64)) as c:
        c.load_files()
        assert np.all(np.isfinite(c.absorption()[0]))
