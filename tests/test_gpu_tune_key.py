"""What the autotuner chose for batches of indexed media is not taken over by
batches of per-cell media of the same size, which run other kernels: they are
tuned by their own steps.  A second batch of the first kind takes no steps."""
import pytest

from mixedprecisionfaracoustic_b200 import Batch
from mixedprecisionfaracoustic_b200.presets import config1

pytestmark = pytest.mark.gpu


def tuned(medium):
    """(steps the autotuner ran, its choice) for a batch of two shots."""
    jobs = [config1(precision="cbf16", nx=n, nz=131, nt=900, npml=11, order=4, nrec=8) for n in (333, 210)]
    for c, _ in jobs:
        c.medium = medium
    b = Batch([c for c, _ in jobs], [m for _, m in jobs])
    try:
        assert (b.medium_tuples(0) > 0) == (medium == "auto")
        t = b.autotune(800)
        return b.cell_updates(), t
    finally:
        b.close()


def test_media_forms_are_tuned_apart():
    first, choice = tuned("auto")
    assert first > 0
    assert tuned("dense")[0] > 0
    again, same = tuned("auto")
    assert again == 0 and same == choice
