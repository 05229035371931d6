"""The safe-haven reducer takes its condition bits a word at a time, split where
the month changes: table lengths around the 32-step words and the four words
loaded together, and months that change inside words, alternate, or are absent.
Whole numbers of steps: every band must equal the oracle exactly."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import products
from test_oracle_lighting_pins import synthetic_horizons

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def session():
    from lunarscout_b200.lightmap_cuda import LightmapCudaSession

    session = LightmapCudaSession(time_batch_size=32)
    yield session
    session.close()


def _months(kind, count):
    if kind == "one":
        return np.zeros(count, np.int32)
    if kind == "blocks":
        return (np.arange(count) // 45 % 5).astype(np.int32)
    if kind == "alternating":
        return (np.arange(count) % 3).astype(np.int32) - 1
    return np.random.default_rng(8).integers(-1, 5, count).astype(np.int32)


@pytest.mark.parametrize("kind", ["one", "blocks", "alternating", "random"])
@pytest.mark.parametrize("count", [1, 31, 32, 33, 127, 128, 129, 301])
def test_every_band_equals_the_oracle(session, count, kind):
    from lunarscout_b200 import synthetic

    hours = synthetic.hours_between("2029-01-20T00", "2029-04-10T00", 3.0)[:count]
    sun, earth = synthetic.sun_vectors(hours), synthetic.earth_vectors(hours)
    dem, horizons = synthetic.config1_dem(), synthetic_horizons()
    tile = dict(tile_y=448, tile_x=448, valid_height=37, valid_width=45)
    fractions = np.stack(list(session.iter_patch_fraction_tiles(dem, horizons, sun, **tile)))
    margins = np.stack(list(session.iter_patch_margin_tiles(dem, horizons, earth, **tile)))
    sunlight, earth_deg = 0.5, float(np.quantile(margins, 0.5))
    months = _months(kind, count)
    got = np.stack(session.safe_haven_durations(
        dem, horizons, sun, earth, month_index_of=months, band_count=5, time_step_hours=3.0,
        sunlight_threshold=sunlight, earth_threshold_deg=earth_deg, **tile))
    expected = products.safe_haven(fractions, margins, months, 5, sunlight_threshold=sunlight,
                                   earth_threshold_deg=earth_deg, time_step_hours=3.0)
    np.testing.assert_array_equal(got, expected)
