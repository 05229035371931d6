"""Vector tables are put in longitude order on the device.  The order only
schedules the steps, so what must hold is that it names every step once: an
ordered launch writes every step's plane, equal to the exact evaluation in time
order.  Lengths around the block's size; longitudes that coincide, straddle
180 degrees, or are not finite."""

from __future__ import annotations

import numpy as np
import pytest

from test_staged_lighting_gpu import _both, _Patch, _vectors

pytestmark = pytest.mark.gpu


def _table(kind, count):
    vectors = _vectors(count, 1.5e11, 700.0)
    if kind == "same":
        vectors[:] = vectors[count // 2]
    elif kind == "seam":
        length = np.linalg.norm(vectors[:, :2], axis=1)
        angle = np.pi + np.linspace(-1e-6, 1e-6, count)
        vectors[:, 0], vectors[:, 1] = length * np.cos(angle), length * np.sin(angle)
        vectors[count // 3, 1] = -0.0
    elif kind == "broken":
        vectors[::7, 0] = np.nan
        vectors[3::11, 1] = np.inf
        vectors[5::13] = 0.0
    return np.ascontiguousarray(vectors, dtype=np.float32)


@pytest.mark.parametrize("kind", ["year", "same", "seam", "broken"])
@pytest.mark.parametrize("count", [1, 31, 1024, 2049])
def test_every_step_is_written_once(cuda_session, count, kind):
    patch = _Patch("walk", width=61, height=50)
    ordered, exact = _both(cuda_session, patch, _table(kind, count), 1)
    np.testing.assert_array_equal(ordered, exact)
