"""Long ordered launches of bodies too near for the staged bounds (within 50
planet radii), wholly or in part of the table, on ragged patches: every output
equals the exact evaluation bit for bit."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from test_staged_lighting_gpu import PLANE, _both, _Patch, _vectors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["smooth", "broken"])
@pytest.mark.parametrize("signal", [0, 1])
@pytest.mark.parametrize("count,far", [(733, 0), (2000, 0), (2000, 300)])
def test_fractions(count, far, signal, kind, cuda_session):
    patch = _Patch(kind, width=119, height=35)
    vectors = _vectors(count, 3.0e7, 8766.0)
    vectors[:far] *= np.float32(1e4)
    got, exact = _both(cuda_session, patch, vectors, signal)
    np.testing.assert_array_equal(got, exact)


@pytest.mark.parametrize("far", [0, 400])
def test_visibility_and_condition_bits(far, cuda_session):
    import torch

    from lunarscout_b200 import _native
    from lunarscout_b200.lightmap_cuda import DeviceVectors

    patch = _Patch("smooth", width=128, height=20)
    vectors = _vectors(1500, 5.0e7, 700.0)
    vectors[:far] *= np.float32(1e3)
    fractions = _both(cuda_session, patch, vectors, 0)[1]
    margins = _both(cuda_session, patch, vectors, 2)[1]
    threshold = float(np.median(margins[:, :20 * 128]))
    visible = torch.empty(PLANE, device="cuda")
    durations = torch.empty((1, PLANE), device="cuda")
    windows, hours = np.array([(0, 1500)], np.int32), np.full(1500, 1.0)
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
                                  (seen.sum(axis=0) / 1500).astype(np.float32)[valid])
    run = longest = np.zeros(PLANE, np.float32)
    for on in seen & (fractions >= np.float32(0.5)):
        run = np.where(on, run + 1, 0)
        longest = np.maximum(longest, run)
    np.testing.assert_array_equal(durations.cpu().numpy()[0, valid],
                                  longest[valid].astype(np.float32))
