"""Segments that the generator does not make, but that a caller of the march may
pass: slopes must equal the CPU oracle's bit for bit, and every ray must end."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from oracle import segments as oseg

pytestmark = pytest.mark.gpu

TILE = dict(tile_column=140, tile_row=140, tile_width=16, subpatch_size=8)
AZIMUTHS = 24


def _case(resolution_m, size=300):
    from lunarscout_b200.contract import PyramidArrays, map_parameters, projection_parameters
    from lunarscout_b200.synthetic import SyntheticDemSpec, synthetic_dem

    dem = synthetic_dem(SyntheticDemSpec(size, resolution_m, latitude_deg=-85.0,
                                         longitude_deg=30.0, craters=20, seed=6))
    mips, levels = oracle.build_pyramid(dem.elevation_m)
    pyramid = PyramidArrays(dem.elevation_m, mips, levels, map_parameters(dem),
                            projection_parameters(dem))
    segments = oseg.build_segments([dem], azimuth_count=AZIMUTHS, maximum_distance_m=9e3,
                                   observer_elevation_m=2.0, **TILE)
    return dem, pyramid, segments


def _expected(segments, pyramid):
    return oracle.march_all_passes(segments, [pyramid], tile_height=16,
                                   observer_elevation_m=2.0, mask=oracle.PRODUCTION_MASK,
                                   **TILE)[0]


def test_device_segments_without_an_end(cuda_session):
    """s_end = +inf: the ray ends where it leaves the DEM.  (One centre has it, so
    that the pixels up and left of it interpolate to it; elsewhere it makes NaN,
    and the ray does not march.)"""
    import torch

    dem, pyramid, segments = _case(20.0)
    segments[:, 10, :, 13] = np.inf
    expected = _expected(segments, pyramid)
    assert np.isfinite(expected[17 * 5]).all() and np.isneginf(expected[17 * 13]).all()
    device = cuda_session.upload_dem_grid(dem)
    device_segments = torch.from_numpy(segments).cuda()
    out = torch.empty((256, AZIMUTHS), device="cuda")
    torch.cuda.synchronize()
    try:
        cuda_session.march_all_passes_device(
            device_segments.data_ptr(), AZIMUTHS, segments.shape[1], [device], tile_height=16,
            observer_elevation_m=2.0, device_out=out.data_ptr(), **TILE)
        cuda_session.synchronize()
    finally:
        device.close()
    np.testing.assert_array_equal(out.cpu().numpy(), expected)


def test_a_path_that_starts_far_behind_its_first_sample(cuda_session):
    """s_start = -3 km: from the first sample on (s = 1 m) the path's offset is
    past 3 km, where a curved path's tangent has little to do with its start."""
    _, pyramid, segments = _case(5.0)
    k1 = segments[..., [4, 8]].copy()  # pixels per km at the sample
    segments[..., [0, 1]] -= k1 * np.float32(3.0 - 9.0 / 6.6)
    segments[..., [2, 3]] = segments[..., [0, 1]]
    segments[..., 4:12] = 0.0
    segments[..., [4, 8]] = k1
    segments[..., [5, 9]] = -k1 / np.float32(6.6)
    segments[..., 12] = -3.0
    segments[..., 16:18] = 0.0
    expected = _expected(segments, pyramid)
    got, _ = cuda_session.subpatch_hierarchical_all_passes(
        segments, [pyramid], tile_height=16, observer_elevation_m=2.0, **TILE)
    assert np.isfinite(expected).mean() > 0.9
    np.testing.assert_array_equal(got, expected)
