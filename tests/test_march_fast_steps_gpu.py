"""The march's settled steps (far_step, level0_step of march_core.cuh) against
the CPU oracle, which takes the reference's full step everywhere: slopes bit
for bit and the same node visits and level-0 samples, on DEMs chosen for the
settled steps' limits: rays along and over the DEM's edges, axis-parallel
rays (tangent components near zero, positions on cell edges), pixels larger
than the angular footprint, invalid cells, running maxima steeper than any
bound, DEMs of a few cells, and one too wide for exact float cell edges."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from oracle import segments as oseg

pytestmark = pytest.mark.gpu


def _dem(height, width, resolution_m, *, longitude_deg=30.0, latitude_deg=-85.0, seed=5,
         sigma_m=150.0):
    from lunarscout_b200.synthetic import SyntheticDemSpec, synthetic_dem

    size = max(64, min(height, width, 512))
    tile = synthetic_dem(SyntheticDemSpec(size, resolution_m, latitude_deg=latitude_deg,
                                          longitude_deg=longitude_deg, sigma_m=sigma_m,
                                          craters=20, seed=seed))
    repeats = (-(-height // size), -(-width // size))
    heights = np.ascontiguousarray(np.tile(tile.elevation_m, repeats)[:height, :width])
    return type(tile)(heights, tile.geo_transform, tile.projection)


def _invalid(dem):
    rng = np.random.default_rng(9)
    for value in (np.nan, np.inf, -np.inf, -25000.0):
        dem.elevation_m.flat[rng.integers(0, dem.elevation_m.size,
                                          size=dem.elevation_m.size // 200)] = value
    return dem


def _walls(dem):
    dem.elevation_m[:, ::7] += 4000.0
    dem.elevation_m[::11, :] -= 3000.0
    return dem


# name -> (DEMs, tile column, row, width, height, azimuths, distance m)
CASES = {
    "inner": lambda: ([_dem(300, 420, 20.0)], 200, 140, 16, 16, 45, 9e3),
    "corner": lambda: ([_dem(300, 420, 20.0)], 0, 0, 16, 16, 48, 9e3),
    "far edge": lambda: ([_dem(301, 423, 10.0)], 416, 290, 16, 16, 37, 9e3),
    "axis": lambda: ([_dem(512, 512, 20.0, longitude_deg=0.0)], 250, 250, 16, 16, 8, 9e3),
    "two passes": lambda: ([_dem(300, 300, 20.0), _dem(500, 400, 240.0, sigma_m=1200.0)],
                           140, 140, 16, 16, 40, 9e4),
    "coarse": lambda: ([_dem(256, 200, 1000.0, sigma_m=900.0)], 100, 90, 16, 16, 40, 1.5e5),
    "fine": lambda: ([_dem(900, 900, 2.0, sigma_m=15.0)], 440, 440, 16, 16, 24, 2000.0),
    "invalid": lambda: ([_invalid(_dem(300, 300, 20.0))], 140, 140, 16, 16, 40, 9e3),
    "walls": lambda: ([_walls(_dem(300, 300, 20.0)), _dem(300, 300, 240.0)],
                      140, 140, 16, 16, 40, 5e4),
    "few cells": lambda: ([_dem(17, 19, 300.0)], 4, 4, 8, 8, 40, 9e4),
    "five rows": lambda: ([_dem(5, 600, 1000.0)], 30, 0, 8, 5, 40, 9e3),
    "too wide": lambda: ([_dem(5, (1 << 22) + 9, 1000.0)], 30, 0, 8, 5, 40, 9e3),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_settled_steps_keep_every_slope_and_decision(name, cuda_session):
    from lunarscout_b200.contract import PyramidArrays, map_parameters, projection_parameters

    dems, column, row, width, height, azimuths, distance = CASES[name]()
    pyramids = []
    for dem in dems:
        mips, levels = oracle.build_pyramid(dem.elevation_m)
        pyramids.append(PyramidArrays(dem.elevation_m, mips, levels, map_parameters(dem),
                                      projection_parameters(dem)))
    tile = dict(tile_column=column, tile_row=row, tile_width=width,
                subpatch_size=2 if dems[0].height < 8 else 8)
    segments = oseg.build_segments(dems, azimuth_count=azimuths, maximum_distance_m=distance,
                                   observer_elevation_m=2.0, **tile)
    tile.update(tile_height=height, observer_elevation_m=2.0)
    gpu, _ = cuda_session.subpatch_hierarchical_all_passes(segments, pyramids, **tile)
    cuda_session.set_counting(True)
    try:
        counted, _ = cuda_session.subpatch_hierarchical_all_passes(segments, pyramids, **tile)
        visits, samples, _ = cuda_session.last_counters()
    finally:
        cuda_session.set_counting(False)
    cpu, expected = oracle.march_all_passes(segments, pyramids, mask=oracle.PRODUCTION_MASK,
                                            **tile)
    np.testing.assert_array_equal(gpu, cpu)
    np.testing.assert_array_equal(counted, cpu)
    assert (visits, samples) == tuple(expected)


@pytest.mark.parametrize("traversal", ["exact", "ladder"])
@pytest.mark.parametrize("name", ["axis", "coarse", "corner", "far edge", "few cells", "fine",
                                  "invalid", "two passes", "walls"])
def test_batched_settled_steps_keep_every_slope_and_decision(name, traversal, cuda_session):
    """The persistent march's steps (ladder_step, march_near among them) on the
    same DEMs: whole tiles of 12 azimuths against the oracle's restatement."""
    import torch

    from lunarscout_b200.contract import PyramidArrays, map_parameters, projection_parameters
    from lunarscout_b200.cuda_backend import SiteTile

    dems, column, row, _, _, _, distance = CASES[name]()
    azimuths = 12
    device = [cuda_session.upload_dem_grid(dem) for dem in dems]
    tile = SiteTile(tuple(device), column, row, distance, 2.0)
    out = torch.empty(128 * 128 * azimuths, device="cuda")
    torch.cuda.synchronize()
    cuda_session.march_sites([tile], device_out=out.data_ptr(), azimuth_count=azimuths,
                             traversal=traversal)
    plain = out.cpu().numpy().reshape(128 * 128, azimuths)
    cuda_session.set_counting(True)
    try:
        cuda_session.march_sites([tile], device_out=out.data_ptr(), azimuth_count=azimuths,
                                 traversal=traversal)
        visits, samples, _ = cuda_session.last_counters()
    finally:
        cuda_session.set_counting(False)
    pyramids = []
    for dem in dems:
        mips, levels = oracle.build_pyramid(dem.elevation_m)
        pyramids.append(PyramidArrays(dem.elevation_m, mips, levels, map_parameters(dem),
                                      projection_parameters(dem)))
    segments = cuda_session.generate_segments(
        device, tile_column=column, tile_row=row, azimuth_count=azimuths,
        maximum_distance_m=distance, observer_elevation_m=2.0)
    mask = oracle.ladder_mask(0, 1) if traversal == "ladder" else oracle.PRODUCTION_MASK
    expected, counts = oracle.march_all_passes(
        segments, pyramids, tile_column=column, tile_row=row, observer_elevation_m=2.0,
        mask=mask)
    np.testing.assert_array_equal(plain, expected)
    np.testing.assert_array_equal(out.cpu().numpy().reshape(expected.shape), expected)
    assert (visits, samples) == tuple(counts)
    for dem in device:
        dem.close()


@pytest.mark.parametrize("height,width", [(4096, 300), (4097, 300), (300, 4097)])
def test_ladder_on_both_sides_of_the_size_limit(height, width, cuda_session):
    """DEMs with a side above 4096 pixels take full steps: the same slopes and
    counters as the oracle's ladder."""
    import torch

    from lunarscout_b200.contract import PyramidArrays, map_parameters, projection_parameters
    from lunarscout_b200.cuda_backend import SiteTile

    dem = _dem(height, width, 5.0)
    column, row, azimuths, distance = min(128, width - 140), 1024 % (height - 130), 8, 30_000.0
    device = cuda_session.upload_dem_grid(dem)
    tile = SiteTile((device,), column, row, distance, 2.0)
    out = torch.empty(128 * 128 * azimuths, device="cuda")
    torch.cuda.synchronize()
    mips, levels = oracle.build_pyramid(dem.elevation_m)
    pyramid = PyramidArrays(dem.elevation_m, mips, levels, map_parameters(dem),
                            projection_parameters(dem))
    segments = cuda_session.generate_segments(
        [device], tile_column=column, tile_row=row, azimuth_count=azimuths,
        maximum_distance_m=distance, observer_elevation_m=2.0)
    expected, counts = oracle.march_all_passes(
        segments, [pyramid], tile_column=column, tile_row=row, observer_elevation_m=2.0,
        mask=oracle.ladder_mask(0, 1))
    for counting in (False, True):
        cuda_session.set_counting(counting)
        try:
            cuda_session.march_sites([tile], device_out=out.data_ptr(), azimuth_count=azimuths,
                                     traversal="ladder")
            counters = cuda_session.last_counters() if counting else None
        finally:
            cuda_session.set_counting(False)
        np.testing.assert_array_equal(out.cpu().numpy().reshape(expected.shape), expected)
    assert counters[:2] == tuple(counts)
    device.close()
