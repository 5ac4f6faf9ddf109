"""Row producers with no output wanted (all four are optional) succeed without
a launch: nothing may be stored through a null row pointer."""

import pytest

from ebsdtorch_b200 import _capi

FAKE = 256  # never dereferenced: nothing is launched
NO_OUTPUT = (None, 0, None, 0, 0, None, None)  # f32, ld, lp, dtype, ld, norm, scale


@pytest.mark.parametrize("n_pix", [63, 64, 6657])
@pytest.mark.parametrize("subtract", [0, 1])
@pytest.mark.parametrize("entry", ["ebsd_project_dictionary", "ebsd_project_dictionary_quads"])
def test_projection_without_outputs(entry, n_pix, subtract):
    assert _capi.call(entry, FAKE, 16, 32, FAKE, n_pix, FAKE, 5, subtract, *NO_OUTPUT, None) in (None, 0)


@pytest.mark.parametrize("h,w", [(7, 9), (8, 8), (129, 129)])
@pytest.mark.parametrize("subtract", [0, 1])
@pytest.mark.parametrize("dtype", [None, 0, 1, 2, 3])
def test_preparation_without_outputs(dtype, h, w, subtract):
    name = "ebsd_prep_patterns" if dtype is None else "ebsd_prep_patterns_typed"
    typed = () if dtype is None else (dtype,)
    assert _capi.call(name, FAKE, *typed, 5, h, w, h * w, 1, None, h * w, subtract, *NO_OUTPUT, None) in (None, 0)


def test_bad_sizes_are_still_refused():
    with pytest.raises(ValueError, match="row length"):
        _capi.call("ebsd_project_dictionary", FAKE, 16, 32, FAKE, 0, FAKE, 5, 1, *NO_OUTPUT, None)
    with pytest.raises(ValueError, match="pattern_stride"):
        _capi.call("ebsd_prep_patterns", FAKE, 5, 8, 8, 63, 1, None, 64, 1, *NO_OUTPUT, None)
