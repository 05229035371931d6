"""The PSR mask of a table is that of its vectors one by one, together: a pixel
is dark when every vector alone leaves it dark.  Launches of one tile and of three
(which take a first look), table lengths around that look and the warp's rounds,
horizons that most, few or no pixels see over, and
vectors that light a pixel only at one place of the table."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from test_staged_batches_gpu import _Tiles
from test_staged_lighting_gpu import PLANE, _Patch, _vectors

pytestmark = pytest.mark.gpu


def _mask(session, patch, vectors, tiles=1):
    """[tiles * 16384] mask of a _Patch or _Tiles."""
    import torch

    from lunarscout_b200 import _native
    from lunarscout_b200.lightmap_cuda import DeviceVectors

    out = torch.full((tiles * PLANE,), 7, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    table = DeviceVectors(session.context, vectors)
    try:
        _native.call("ls200_lighting_device", session.context, *patch.args(), table.handle, 0,
                     len(vectors), 3, ctypes.c_void_p(patch.frames.data_ptr()),
                     ctypes.c_void_p(out.data_ptr()))
        session.synchronize()
    finally:
        table.close()
    return out.cpu().numpy()


@pytest.mark.parametrize("kind", ["smooth", "steep", "broken"])
@pytest.mark.parametrize("count", [1, 2, 3, 4, 5, 7, 8, 9, 31, 32, 33, 65, 130])
def test_a_table_is_its_vectors_together(count, kind, cuda_session):
    patch = _Patch(kind, width=101, height=77, seed=count)
    vectors = _vectors(count, 1.5e11, 8766.0)
    singles = [_mask(cuda_session, patch, vectors[t:t + 1]) for t in range(count)]
    got = _mask(cuda_session, patch, vectors)
    np.testing.assert_array_equal(got, np.minimum.reduce(singles))
    valid = (np.arange(PLANE) % 128 < 101) & (np.arange(PLANE) // 128 < 77)
    assert set(np.unique(got[valid])) <= {0, 255} and not got[~valid].any()


@pytest.mark.parametrize("place", [0, 1, 2, 24, 25, 50, 75, 98, 99])
def test_one_vector_lights_the_pixels(place, cuda_session):
    patch = _Patch("smooth")
    vectors = np.repeat(np.array([[0.0, 0.0, 1.5e11]], np.float32), 100, axis=0)  # below
    assert (_mask(cuda_session, patch, vectors) == 255).all()
    vectors[place] = _vectors(1, 1.5e11, 0.0)[0] + np.float32([0.0, 0.0, -5e10])
    alone = _mask(cuda_session, patch, vectors[place:place + 1])
    assert (alone == 0).any()
    np.testing.assert_array_equal(_mask(cuda_session, patch, vectors), alone)


@pytest.mark.parametrize("count", [1, 2, 3, 15, 16, 17, 18, 32, 33, 64, 100])
def test_three_tiles_are_their_vectors_together(count, cuda_session):
    tiles, vectors = _Tiles(), _vectors(count, 1.5e11, 8766.0)
    singles = [_mask(cuda_session, tiles, vectors[t:t + 1], 3) for t in range(count)]
    got = _mask(cuda_session, tiles, vectors, 3)
    np.testing.assert_array_equal(got, np.minimum.reduce(singles))
    for i in range(3):
        part = got[i * PLANE:(i + 1) * PLANE]
        assert not part[~tiles.valid(i)].any()
        # The same tile alone takes no first look.
        patch = _Patch("flat")
        patch.horizons, patch.dem = tiles.horizons[i].reshape(-1), tiles.dems[i]
        patch.window = tiles.windows[i].copy()
        np.testing.assert_array_equal(part, _mask(cuda_session, patch, vectors))


@pytest.mark.parametrize("place", [0, 1, 24, 50, 51, 98, 99])
def test_one_vector_lights_three_tiles(place, cuda_session):
    tiles = _Tiles()
    vectors = np.repeat(np.array([[0.0, 0.0, 1.5e11]], np.float32), 100, axis=0)
    vectors[place] = _vectors(1, 1.5e11, 0.0)[0] + np.float32([0.0, 0.0, -5e10])
    alone = _mask(cuda_session, tiles, vectors[place:place + 1], 3)
    assert (alone == 0).any() and (alone == 255).any()
    below = _mask(cuda_session, tiles, vectors[(place + 1) % 100:][:1], 3)
    np.testing.assert_array_equal(_mask(cuda_session, tiles, vectors, 3),
                                  np.minimum(alone, below))
