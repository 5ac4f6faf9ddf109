"""Which detectors' correlation reads quads: those of the tensor-memory kernel."""

import pytest

from ebsdtorch_b200.ebsd import fitting


@pytest.mark.parametrize("hp,wp,suffix", [(2, 2, "_quads"), (23, 22, "_quads"), (78, 78, "_quads"),
                                          (96, 96, "_quads"), (127, 64, "_quads"), (97, 97, ""), (104, 104, ""),
                                          (64, 127, ""), (127, 127, ""), (128, 64, "")])
def test_layout_of_a_detector(hp, wp, suffix):
    assert fitting.spectra_layout(hp, wp) == suffix
