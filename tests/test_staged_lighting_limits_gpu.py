"""Where the staged lighting's approximate direction is poor, samples must take
the exact one: bodies near the zenith and the nadir, whose azimuth hangs on the
rounding of the vector, and vectors so long that their squares overflow.  The
entry without an order evaluates every sample exactly; outputs must equal its
bit for bit."""

from __future__ import annotations

import numpy as np
import pytest

from test_staged_lighting_gpu import AZ, PLANE, _both, _Patch, _vectors

pytestmark = pytest.mark.gpu


def _near_vertical(session, patch, sign, count=1200):
    """Vectors 1e-6 to 1e-2 rad from the vertical of a patch of 1 cm pixels, in
    a few degrees of azimuth, after giving it horizons of bins that block every
    body (or, below, let it pass) in turn with flat ones."""
    import torch

    patch.geo[[1, 5]] = 0.01, -0.01
    _both(session, patch, _vectors(2, 1.5e11, 10.0), 0)
    frame = patch.frames.cpu().numpy().reshape(PLANE, 12)[64 * 128 + 64].astype(np.float64)
    east, north, up = frame[[0, 3, 6]], frame[[1, 4, 7]], frame[[2, 5, 8]]
    rng = np.random.default_rng(7)
    tilt = 10.0 ** rng.uniform(-6.0, -2.0, (count, 1))
    azimuth = rng.uniform(0.5, 0.55, (count, 1))
    rows = np.where(rng.integers(0, 2, (PLANE, AZ // 12)) > 0, sign * 5e4, 0.0)
    patch.horizons.copy_(torch.from_numpy(np.repeat(rows, 12, axis=1).astype("f4").reshape(-1)))
    vectors = sign * up + tilt * (np.sin(azimuth) * east + np.cos(azimuth) * north)
    return np.ascontiguousarray(1.5e11 * vectors, dtype=np.float32)


@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("signal", [0, 1])
def test_bodies_near_the_vertical(sign, signal, cuda_session):
    patch = _Patch("flat")
    vectors = _near_vertical(cuda_session, patch, sign)
    got, exact = _both(cuda_session, patch, vectors, signal)
    assert (exact != exact.flat[0]).any()
    np.testing.assert_array_equal(got, exact)


@pytest.mark.parametrize("scale", [1e9, 1e12, 1e26])
def test_vectors_of_mixed_length(scale, cuda_session):
    """1.5e37 m still fits a float; from 1.8e19 m on the squares do not."""
    patch = _Patch("smooth")
    vectors = _vectors(1100, 1.5e11, 8766.0)
    vectors[::9] *= np.float32(scale)
    assert np.isfinite(vectors).all()
    got, exact = _both(cuda_session, patch, vectors, 1)
    np.testing.assert_array_equal(got, exact)
