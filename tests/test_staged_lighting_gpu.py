"""Long ordered lighting launches (staged_samples of lighting.cu) settle clear
samples from bounds; every output must equal the exact evaluation bit for bit.
The allocation-free entry evaluates every sample exactly (it has no order), so
it is the reference here.  Cases: table lengths around the staging limit and
chunk sizes, ragged patches, horizons with steep, infinite and NaN bins, the
body near azimuth 0, bodies too near for the bounds, thresholds at the signals'
ends, and misaligned device arrays."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PLANE, AZ = 128 * 128, 1440


def _horizons(kind, rng):
    rows = rng.normal(0.0, 0.3, size=(PLANE, AZ)).cumsum(axis=1).astype(np.float32)
    rows = rows / np.float32(8.0) + rng.normal(0.0, 1.5, size=(PLANE, 1)).astype(np.float32)
    if kind == "steep":
        rows[:, ::5] += rng.choice((-30.0, 20.0, 60.0, 85.0), size=(PLANE, AZ // 5)).astype("f4")
    elif kind == "broken":
        spots = rng.integers(0, rows.size, size=rows.size // 40)
        rows.flat[spots] = rng.choice((np.inf, -np.inf, np.nan, -50.0, 90.0, 1e30),
                                      size=len(spots)).astype("f4")
    elif kind == "flat":
        rows[:] = 0.0
    return np.ascontiguousarray(rows)


class _Patch:
    def __init__(self, kind, *, width=128, height=128, shift=0, seed=3, y=151_000.0):
        import torch

        rng = np.random.default_rng(seed)
        rows = _horizons(kind, rng)
        # `shift` floats into the allocation: a misaligned device array.
        self.horizons = torch.empty(rows.size + shift, device="cuda")[shift:]
        self.horizons.copy_(torch.from_numpy(rows.reshape(-1)))
        self.dem = torch.from_numpy(rng.normal(0, 300, PLANE).astype("f4")).cuda()
        self.geo = np.array((12_000.0, 20.0, 0.0, y, 0.0, -20.0))
        self.projection = np.array((1_737_400.0, -np.pi / 2, 0.0, 1.0, 0.0, 0.0))
        self.window = np.array((5, 9, width, height), np.int32)
        self.frames = torch.empty(PLANE * 12 + shift, device="cuda")[shift:]

    def args(self):
        return (1, ctypes.c_void_p(self.dem.data_ptr()), self.geo.ctypes.data,
                self.projection.ctypes.data, self.window.ctypes.data,
                ctypes.c_void_p(self.horizons.data_ptr()))


def _vectors(count, distance_m, hours):
    from lunarscout_b200 import synthetic

    sun = synthetic.sun_vectors(np.linspace(0.0, hours, count))
    return np.ascontiguousarray(sun * (distance_m / np.linalg.norm(sun[0])), dtype=np.float32)


def _both(session, patch, vectors, signal):
    """(ordered launch, exact launch) of a signal, [T, 16384]."""
    import torch

    from lunarscout_b200 import _native
    from lunarscout_b200.lightmap_cuda import DeviceVectors

    dtype = torch.uint8 if signal == 1 else torch.float32
    out = [torch.full((len(vectors), PLANE), 7, dtype=dtype, device="cuda") for _ in range(2)]
    device_vectors = torch.from_numpy(vectors).cuda()
    torch.cuda.synchronize()
    table = DeviceVectors(session.context, vectors)
    try:
        _native.call("ls200_lighting_device", session.context, *patch.args(), table.handle, 0,
                     len(vectors), signal, ctypes.c_void_p(patch.frames.data_ptr()),
                     ctypes.c_void_p(out[0].data_ptr()))
        _native.call("ls200_lighting_device_noalloc", session.context, *patch.args(),
                     ctypes.c_void_p(device_vectors.data_ptr()), len(vectors), 0, len(vectors),
                     signal, ctypes.c_void_p(out[1].data_ptr()))
        session.synchronize()
    finally:
        table.close()
    return [o.cpu().numpy() for o in out]


CASES = [("smooth", dict(), 719), ("smooth", dict(), 720), ("smooth", dict(width=77, height=3), 1001),
         ("steep", dict(), 1500), ("broken", dict(), 1441), ("flat", dict(), 900),
         ("smooth", dict(shift=1), 1200), ("steep", dict(width=1, height=128, shift=2), 3001),
         ("steep", dict(y=931_000.0), 1800)]


@pytest.mark.parametrize("kind,options,count", CASES)
@pytest.mark.parametrize("signal", [0, 1])
def test_settled_fractions_equal_the_exact_ones(kind, options, count, signal, cuda_session):
    got, exact = _both(cuda_session, _Patch(kind, **options), _vectors(count, 1.5e11, 8766.0),
                       signal)
    np.testing.assert_array_equal(got, exact)
    assert (exact != exact.flat[0]).any()


@pytest.mark.parametrize("distance_m", [1.8e6, 2e7, 8.7e7, 3.8e8])
def test_bodies_of_any_distance(distance_m, cuda_session):
    got, exact = _both(cuda_session, _Patch("smooth"), _vectors(800, distance_m, 700.0), 0)
    np.testing.assert_array_equal(got, exact)


@pytest.mark.parametrize("kind", ["smooth", "steep", "broken"])
@pytest.mark.parametrize("threshold,y", [(0.0, 151e3), (2.0, 151e3), (-4.5, 151e3),
                                         (25.0, 931e3), (-60.0, 931e3), (95.0, 931e3)])
def test_visibility_counts_the_exact_margins(kind, threshold, y, cuda_session):
    import torch

    from lunarscout_b200 import _native
    from lunarscout_b200.lightmap_cuda import DeviceVectors

    patch = _Patch(kind, width=128, height=90, y=y)  # y: latitude -85 or -60
    vectors = _vectors(1300, 3.8e8, 8766.0)
    _, margins = _both(cuda_session, patch, vectors, 2)
    out = torch.empty(PLANE, device="cuda")
    torch.cuda.synchronize()
    table = DeviceVectors(cuda_session.context, vectors)
    try:
        _native.call("ls200_earth_visibility_device", cuda_session.context, *patch.args(),
                     table.handle, float(threshold), ctypes.c_void_p(out.data_ptr()))
    finally:
        table.close()
    expected = ((margins >= np.float32(threshold)).sum(axis=0) / len(vectors)).astype(np.float32)
    got = out.cpu().numpy().reshape(128, 128)
    np.testing.assert_array_equal(got[:90], expected.reshape(128, 128)[:90])
    assert np.isnan(got[90:]).all()


@pytest.mark.parametrize("sun_threshold", [0.0, 0.2, 0.5, 1.0])
def test_condition_bits_and_their_runs(sun_threshold, cuda_session):
    """Longest runs per window from the staged bits, against runs counted on
    the exact signals."""
    import torch

    from lunarscout_b200 import _native
    from lunarscout_b200.lightmap_cuda import DeviceVectors

    patch = _Patch("smooth", width=128, height=20)
    sun, earth = _vectors(1700, 1.5e11, 8766.0), _vectors(1700, 3.8e8, 7000.0)
    windows = np.array([(0, 1700), (0, 0), (100, 133), (1650, 1700), (64, 65), (31, 1000)],
                       np.int32)
    on = (_both(cuda_session, patch, sun, 0)[1] >= np.float32(sun_threshold)) & (
        _both(cuda_session, patch, earth, 2)[1] >= np.float32(0.5))
    out = torch.empty((len(windows), PLANE), device="cuda")
    torch.cuda.synchronize()
    hours = np.full(len(sun), 1.0)
    tables = [DeviceVectors(cuda_session.context, v) for v in (sun, earth)]
    try:
        _native.call("ls200_mission_duration_device", cuda_session.context, *patch.args(),
                     tables[0].handle, tables[1].handle, float(sun_threshold), 0.5,
                     hours.ctypes.data, windows.ctypes.data, len(windows), 0,
                     ctypes.c_void_p(out.data_ptr()))
    finally:
        for table in tables:
            table.close()
    got = out.cpu().numpy()
    expected = np.zeros((len(windows), PLANE), np.float32)
    start = np.full(PLANE, -1)
    for t in range(len(sun)):
        start = np.where(on[t], np.where(start < 0, t, start), -1)
        for i, (first, end) in enumerate(windows):
            begin = np.maximum(start, first)
            live = on[t] & (begin < end) & (begin <= t)
            expected[i] = np.where(live, np.maximum(expected[i], t + 1 - begin), expected[i])
    valid = np.arange(PLANE) < 20 * 128
    np.testing.assert_array_equal(got[:, valid], expected[:, valid])
    assert not got[:, ~valid].any()
