"""Staged lighting launches over several tiles and over a part of a vector
table, and the products made of their bits, against the exact evaluation (the
entry without an order) of the same tiles: a wrong tile or time offset, or a
condition the wrong way round, shows in any of them."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from oracle import products
from test_staged_lighting_gpu import AZ, PLANE, _horizons, _vectors

pytestmark = pytest.mark.gpu

WINDOWS = np.array([(5, 9, 128, 128), (133, 9, 128, 41), (5, 137, 77, 128)], np.int32)


class _Tiles:
    def __init__(self, kinds=("smooth", "steep", "broken")):
        import torch

        rng = np.random.default_rng(12)
        self.count = len(kinds)
        self.horizons = torch.empty((self.count, PLANE, AZ), device="cuda")
        for i, kind in enumerate(kinds):
            self.horizons[i] = torch.from_numpy(_horizons(kind, rng))
        self.dems = torch.from_numpy(rng.normal(0, 300, (self.count, PLANE)).astype("f4")).cuda()
        self.geo = np.repeat([(12_000.0, 20.0, 0.0, 151_000.0, 0.0, -20.0)], self.count, 0)
        self.projection = np.repeat([(1_737_400.0, -np.pi / 2, 0.0, 1.0, 0.0, 0.0)], self.count, 0)
        self.windows = WINDOWS[:self.count].copy()
        self.frames = torch.empty(self.count * PLANE * 12, device="cuda")

    def args(self):
        return (self.count, ctypes.c_void_p(self.dems.data_ptr()), self.geo.ctypes.data,
                self.projection.ctypes.data, self.windows.ctypes.data,
                ctypes.c_void_p(self.horizons.data_ptr()))

    def valid(self, i):
        width, height = self.windows[i, 2:]
        index = np.arange(PLANE)
        return (index % 128 < width) & (index // 128 < height)


def _call(session, tiles, vectors, signal, start, count, ordered):
    """Signal planes [n, count, 16384] of steps [start, start + count)."""
    import torch

    from lunarscout_b200 import _native
    from lunarscout_b200.lightmap_cuda import DeviceVectors

    out = torch.full((tiles.count, count, PLANE), 7, device="cuda",
                     dtype=torch.uint8 if signal == 1 else torch.float32)
    on_device = torch.from_numpy(vectors).cuda()
    torch.cuda.synchronize()
    table = DeviceVectors(session.context, vectors)
    try:
        if ordered:
            _native.call("ls200_lighting_device", session.context, *tiles.args(), table.handle,
                         start, count, signal, ctypes.c_void_p(tiles.frames.data_ptr()),
                         ctypes.c_void_p(out.data_ptr()))
        else:
            _native.call("ls200_lighting_device_noalloc", session.context, *tiles.args(),
                         ctypes.c_void_p(on_device.data_ptr()), len(vectors), start, count,
                         signal, ctypes.c_void_p(out.data_ptr()))
        session.synchronize()
    finally:
        table.close()
    return out.cpu().numpy()


@pytest.mark.parametrize("signal", [0, 1, 2])
@pytest.mark.parametrize("start,count", [(0, 1900), (341, 1100), (1177, 723), (1200, 300)])
def test_several_tiles_and_a_part_of_the_table(start, count, signal, cuda_session):
    tiles, vectors = _Tiles(), _vectors(1900, 1.5e11, 8766.0)
    got = _call(cuda_session, tiles, vectors, signal, start, count, True)
    exact = _call(cuda_session, tiles, vectors, signal, start, count, False)
    np.testing.assert_array_equal(got, exact)


@pytest.mark.parametrize("threshold", [0.0, -3.0])
def test_visibility_of_several_tiles(threshold, cuda_session):
    import torch

    from lunarscout_b200 import _native
    from lunarscout_b200.lightmap_cuda import DeviceVectors

    tiles, vectors = _Tiles(), _vectors(1300, 3.8e8, 8766.0)
    margins = _call(cuda_session, tiles, vectors, 2, 0, len(vectors), False)
    out = torch.empty((tiles.count, PLANE), device="cuda")
    torch.cuda.synchronize()
    table = DeviceVectors(cuda_session.context, vectors)
    try:
        _native.call("ls200_earth_visibility_device", cuda_session.context, *tiles.args(),
                     table.handle, threshold, ctypes.c_void_p(out.data_ptr()))
    finally:
        table.close()
    got = out.cpu().numpy()
    expected = ((margins >= np.float32(threshold)).sum(axis=1) / len(vectors)).astype("f4")
    for i in range(tiles.count):
        valid = tiles.valid(i)
        np.testing.assert_array_equal(got[i, valid], expected[i, valid])
        assert np.isnan(got[i, ~valid]).all()


@pytest.mark.parametrize("sunlight,earth_deg", [(0.0, 2.0), (0.2, 2.0), (1.0, -3.5), (0.5, 0.0)])
def test_safe_haven_of_a_long_table(sunlight, earth_deg, cuda_session):
    """1,700 steps: both condition planes are staged, as `below a threshold`."""
    import torch

    from lunarscout_b200 import _native
    from lunarscout_b200.lightmap_cuda import DeviceVectors

    tiles = _Tiles(("smooth", "steep"))
    sun, earth = _vectors(1700, 1.5e11, 8766.0), _vectors(1700, 3.8e8, 7000.0)
    months = (np.arange(1700) // 150).astype(np.int32)
    bands = int(months[-1]) + 1
    out = torch.empty((tiles.count, bands, PLANE), device="cuda")
    torch.cuda.synchronize()
    tables = [DeviceVectors(cuda_session.context, v) for v in (sun, earth)]
    try:
        _native.call("ls200_safe_haven_device", cuda_session.context, *tiles.args(),
                     tables[0].handle, tables[1].handle, sunlight, earth_deg, 2.0,
                     months.ctypes.data, bands, ctypes.c_void_p(out.data_ptr()))
    finally:
        for table in tables:
            table.close()
    got = out.cpu().numpy()
    fractions = _call(cuda_session, tiles, sun, 0, 0, 1700, False)
    margins = _call(cuda_session, tiles, earth, 2, 0, 1700, False)
    for i in range(tiles.count):
        pixels = np.flatnonzero(tiles.valid(i))[::97]
        expected = products.safe_haven(
            fractions[i][:, None, pixels], margins[i][:, None, pixels], months, bands,
            sunlight_threshold=sunlight, earth_threshold_deg=earth_deg, time_step_hours=2.0)
        np.testing.assert_array_equal(got[i][:, pixels], np.asarray(expected)[:, 0])


@pytest.mark.parametrize("sun_threshold", [0.2, 1.0])
def test_mission_duration_of_several_tiles(sun_threshold, cuda_session):
    import torch

    from lunarscout_b200 import _native
    from lunarscout_b200.lightmap_cuda import DeviceVectors

    tiles = _Tiles()
    sun, earth = _vectors(1500, 1.5e11, 8766.0), _vectors(1500, 3.8e8, 7000.0)
    on = (_call(cuda_session, tiles, sun, 0, 0, 1500, False) >= np.float32(sun_threshold)) & (
        _call(cuda_session, tiles, earth, 2, 0, 1500, False) >= np.float32(0.5))
    windows = np.array([(0, 1500)], np.int32)
    out = torch.empty((tiles.count, 1, PLANE), device="cuda")
    torch.cuda.synchronize()
    hours = np.full(1500, 1.0)
    tables = [DeviceVectors(cuda_session.context, v) for v in (sun, earth)]
    try:
        _native.call("ls200_mission_duration_device", cuda_session.context, *tiles.args(),
                     tables[0].handle, tables[1].handle, sun_threshold, 0.5, hours.ctypes.data,
                     windows.ctypes.data, 1, 0, ctypes.c_void_p(out.data_ptr()))
    finally:
        for table in tables:
            table.close()
    got = out.cpu().numpy()
    run = np.zeros((tiles.count, PLANE), np.float32)
    longest = run.copy()
    for t in range(1500):
        run = np.where(on[:, t], run + 1, 0)
        longest = np.maximum(longest, run)
    for i in range(tiles.count):
        valid = tiles.valid(i)
        np.testing.assert_array_equal(got[i, 0, valid], longest[i, valid])
