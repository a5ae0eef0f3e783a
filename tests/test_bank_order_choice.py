"""Which Trotter jobs get the warp kernels' bank order (host only): every one whose
rotations run on those kernels, a tuned job on the kernel that the tuner chose, as
the tuner timed it with the order."""
import pytest

import nise_2017_b200 as nise


@pytest.mark.parametrize("forced, tuned, rows, autotune, order", [
    (0, None, 0, 0, 1), (0, None, 35, 0, 0), (0, None, 36, 0, 0),   # untuned: by the default
    (0, 32, 35, 0, 1), (0, 34, 36, 0, 1), (0, 0, 35, 0, 1),         # tuned to another kernel than the default rows
    (0, 35, 0, 0, 0), (0, 36, 35, 0, 0), (0, 33, 0, 0, 1),
    (0, None, 35, 1, 1), (0, 35, 35, 1, 1),                         # the tuner times both
    (35, None, 35, 0, 0), (36, 32, 0, 1, 0), (32, 35, 0, 0, 1), (1, None, 0, 0, 1)])
def test_bank_order_choice(forced, tuned, rows, autotune, order):
    call = nise.lib().nise_trotter_needs_bank_order
    assert call(forced, int(tuned is not None), tuned or 0, rows, autotune) == order
