"""Small segment launches give each job 16 lanes; large ones a thread.  Every
field must be the same bit for bit.  A subpatch centre of a small tile is also a
centre of a large tile around it, so each case generates both and compares the
centres that they share: rays that end inside the DEM and that leave it, short
rays, tiles at the DEM's edges, a coarse second DEM, and pole-side sites."""

from __future__ import annotations

import numpy as np
import pytest

from lunarscout_b200.synthetic import SyntheticDemSpec, synthetic_dem

pytestmark = pytest.mark.gpu

SMALL, LARGE, STEP = 16, 128, 8


def _site(side, resolution, latitude=-88.5):
    return synthetic_dem(SyntheticDemSpec(side, resolution, latitude_deg=latitude,
                                          longitude_deg=30.0, seed=5))


CASES = {
    "inside": (lambda: [_site(400, 20.0)], 136, 144, 500.0, 120),
    "leaving": (lambda: [_site(300, 20.0)], 136, 96, 50_000.0, 119),
    "corner": (lambda: [_site(300, 5.0)], 0, 0, 4_000.0, 97),
    "far corner": (lambda: [_site(260, 5.0)], 232, 240, 4_000.0, 97),
    "two": (lambda: [_site(300, 5.0), _site(500, 240.0)], 128, 120, 100_000.0, 73),
    "short": (lambda: [_site(300, 20.0)], 128, 128, 1.3, 121),
    "few metres": (lambda: [_site(300, 1.0)], 128, 128, 60.0, 60),
    "polar": (lambda: [_site(300, 20.0, -89.99)], 128, 128, 20_000.0, 64),
}


@pytest.mark.parametrize("name", list(CASES))
def test_both_launches_give_the_same_segments(name, cuda_session):
    make, column, row, distance, azimuths = CASES[name]
    dems = [cuda_session.upload_dem_grid(dem) for dem in make()]
    try:
        options = dict(azimuth_count=azimuths, maximum_distance_m=distance,
                       observer_elevation_m=2.0, subpatch_size=STEP)
        small = cuda_session.generate_segments(dems, tile_column=column, tile_row=row,
                                               tile_width=SMALL, **options)
        left, top = max(0, column - 48), max(0, row - 56)
        large = cuda_session.generate_segments(dems, tile_column=left, tile_row=top,
                                               tile_width=LARGE, **options)
    finally:
        for dem in dems:
            dem.close()
    count = SMALL // STEP + 2
    wide = LARGE // STEP + 2
    index = np.arange(count)
    shared = ((index[:, None] + (row - top) // STEP) * wide + index + (column - left) // STEP)
    assert small.shape[1] * azimuths <= 6144 < large.shape[1] * azimuths
    np.testing.assert_array_equal(small.view(np.uint32),
                                  large[:, shared.ravel()].view(np.uint32))
