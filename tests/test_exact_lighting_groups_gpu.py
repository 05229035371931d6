"""Exact lighting launches (short tables, and rows that cannot be staged) take
their steps in small chunks, or a group of chunks at once with the bins in a
window where the group's bodies lie close together.  Either way every step is
evaluated once and equals the entry without an order bit for bit: table lengths
around the chunks and groups, arcs from one direction to the whole circle, and
bodies whose azimuth at the pixel does not follow their longitude."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from test_staged_lighting_gpu import PLANE, _both, _Patch, _vectors

pytestmark = pytest.mark.gpu

HOURS = {"one": 0.0, "hour": 1.0, "day": 24.0, "five days": 120.0, "ten days": 240.0,
         "year": 8766.0}


@pytest.mark.parametrize("arc", list(HOURS))
@pytest.mark.parametrize("count", [1, 3, 16, 17, 68, 125, 355, 719])
@pytest.mark.parametrize("signal", [0, 2])
def test_every_step_equals_the_exact_entry(count, arc, signal, cuda_session):
    patch = _Patch("steep", width=109, height=33)
    got, exact = _both(cuda_session, patch, _vectors(count, 1.5e11, HOURS[arc]), signal)
    np.testing.assert_array_equal(got, exact)


@pytest.mark.parametrize("arc", ["day", "year"])
@pytest.mark.parametrize("signal", [0, 1, 2])
def test_misaligned_rows_of_a_long_table(arc, signal, cuda_session):
    patch = _Patch("broken", width=128, height=20, shift=1)
    got, exact = _both(cuda_session, patch, _vectors(2000, 1.5e11, HOURS[arc]), signal)
    np.testing.assert_array_equal(got, exact)


@pytest.mark.parametrize("y", [151_000.0, 1_500_000.0])
@pytest.mark.parametrize("signal", [0, 2])
def test_near_and_far_latitudes_with_broken_vectors(y, signal, cuda_session):
    patch = _Patch("broken", width=64, height=64, y=y)
    vectors = _vectors(400, 1.5e11, 120.0)
    vectors[::31, 0] = np.nan
    vectors[5::47] = 0.0
    got, exact = _both(cuda_session, patch, vectors, signal)
    np.testing.assert_array_equal(got, exact)


@pytest.mark.parametrize("arc", ["hour", "ten days", "year"])
@pytest.mark.parametrize("count", [33, 400])
def test_visibility_and_condition_bits(count, arc, cuda_session):
    import torch

    from lunarscout_b200 import _native
    from lunarscout_b200.lightmap_cuda import DeviceVectors

    patch = _Patch("smooth", width=128, height=20)
    vectors = _vectors(count, 3.8e8, HOURS[arc])
    fractions = _both(cuda_session, patch, vectors, 0)[1]
    margins = _both(cuda_session, patch, vectors, 2)[1]
    threshold = float(np.median(margins[:, :20 * 128]))
    visible = torch.empty(PLANE, device="cuda")
    durations = torch.empty((1, PLANE), device="cuda")
    windows, hours = np.array([(0, count)], np.int32), np.full(count, 1.0)
    torch.cuda.synchronize()
    table = DeviceVectors(cuda_session.context, vectors)
    try:
        _native.call("ls200_earth_visibility_device", cuda_session.context, *patch.args(),
                     table.handle, threshold, ctypes.c_void_p(visible.data_ptr()))
        _native.call("ls200_mission_duration_device", cuda_session.context, *patch.args(),
                     table.handle, table.handle, 0.5, threshold, hours.ctypes.data,
                     windows.ctypes.data, 1, 0, ctypes.c_void_p(durations.data_ptr()))
    finally:
        table.close()
    valid = np.arange(PLANE) < 20 * 128
    seen = margins >= np.float32(threshold)
    np.testing.assert_array_equal(visible.cpu().numpy()[valid],
                                  (seen.sum(axis=0) / count).astype(np.float32)[valid])
    run = longest = np.zeros(PLANE, np.float32)
    for on in seen & (fractions >= np.float32(0.5)):
        run = np.where(on, run + 1, 0)
        longest = np.maximum(longest, run)
    np.testing.assert_array_equal(durations.cpu().numpy()[0, valid],
                                  longest[valid].astype(np.float32))
