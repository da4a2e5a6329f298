"""The raster passes' packed division: a small triangle's pixel q of a bounding box w wide lies in row q / w, taken as
q * inv >> 15 with inv = floor(2^15 / w) + 1, or one more (an approximate quotient may round up)."""
import numpy as np
import pytest


@pytest.mark.parametrize("extra", [1, 2])
def test_packed_division_is_exact(extra):
    q, w = np.meshgrid(np.arange(128), np.arange(1, 129), indexing="ij")
    inv = (1 << 15) // w + extra
    assert (inv < 1 << 16).all()
    assert np.array_equal((q * inv) >> 15, q // w)


@pytest.mark.parametrize("extra", [0, 1, 2])
def test_box_steps_are_exact(extra):
    """warp_draw's quotients of a lane and of 32 pixels by a box width, whichever way the reciprocal rounds."""
    lane, w = np.meshgrid(np.arange(33), np.arange(1, 32769), indexing="ij")
    inv = (1 << 15) // w + extra
    if extra == 0:  # an approximate quotient falls below the exact one only where that is whole
        lane, w, inv = (a[:, (1 << 15) % w[0] == 0] for a in (lane, w, inv))
    assert np.array_equal((lane * inv) >> 15, lane // w)
