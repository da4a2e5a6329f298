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
