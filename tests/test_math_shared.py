"""The elementary functions evaluated side by side (sc_sincosf, sc_sin3 of
spatial_cell_gb300/csrc/scmath.h) give the bits of the single ones: over every
exponent, on signed zeros, infinities and NaN, and where one of three
arguments leaves the range they are reduced together in."""
import numpy as np
import pytest

from tests.test_math import _eval, lib  # noqa: F401


def _bits(a):
    return np.where(np.isnan(a), np.uint32(0x7fc00000), a.view(np.uint32))


@pytest.mark.parametrize("joint,single,flip", [(6, 0, False), (7, 1, False), (8, 0, False), (9, 0, True)])
def test_same_bits(lib, joint, single, flip):  # noqa: F811
    rng = np.random.default_rng(joint)
    x = rng.integers(0, 1 << 32, 300000, np.uint64).astype(np.uint32).view(np.float32)
    x = np.concatenate([x, rng.uniform(-8, 8, 300000).astype(np.float32),
                        np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1000.0, 1000.1, -1000.1], np.float32)])
    y = rng.permutation(x)
    assert np.array_equal(_bits(_eval(lib, joint, x, y)), _bits(_eval(lib, single, -x if flip else x)))
