"""Performance cases of the horizon and lighting path.

Each case is one call (or the pair of calls a program always makes together)
of the public entry points, on seeded synthetic inputs: fBm terrain with
craters on a south-polar grid, 1440-azimuth horizon tiles of such terrain, and
Sun / Earth vectors of the lunar motion.  Sizes are those of the benchmark,
the tests and the tile generator, with ragged and small ones between them.

Kinds:
  tile        segments + every DEM pass of one tile, on the device
              (CudaSession.generate_segments_device, march_all_passes_device)
  session     the host drop-in CudaSession.subpatch_hierarchical_all_passes
  sites       tiles of several sites in one persistent launch
              (CudaSession.march_sites)
  lightmap    ProductChain.sun_fractions / sun_fraction_bytes
  psr         ProductChain.psr with the device vector reduction
  mission     ProductChain.mission_durations
  haven       ProductChain.safe_haven
  visibility  ProductChain.earth_visibility
  codec       TileCodec.encode_device / decode of one tile
  adjoint     SunLossProblem: new heights, loss and gradients
"""

from __future__ import annotations

import math

import numpy as np
import torch

from lunarscout_b200.chain import PatchBatch, ProductChain
from lunarscout_b200.contract import DemGrid, ProjectionParameters
from lunarscout_b200.cuda_backend import CudaSession, SiteTile
from lunarscout_b200.file_format import MAX_PAYLOAD_BYTES, TileCodec
from lunarscout_b200.pipeline import PatchDescriptor

RADIUS_M = 1_737_400.0
AU_M = 149_597_870_700.0
EARTH_M = 384_400_000.0
SIDE = 128
PLANE = SIDE * SIDE
AZIMUTHS = 1440
SUBPATCH = 8


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # A quick look at a few pixels of a small DEM (an interactive preview,
        # a unit test): launches and latency count, not throughput.
        {"name": "tile-preview", "kind": "tile", "height": 200, "width": 256,
         "resolution_m": 20.0, "regional": False, "distance_m": 5_000.0, "tile_x": 96,
         "tile_y": 64, "tile_w": 16, "tile_h": 16, "azimuths": 72, "degrees": True},
        # The plain configuration of the tests: one tile of a 512 x 512 DEM at
        # 20 m, rays of 10 km, every azimuth.
        {"name": "tile-plain", "kind": "tile", "height": 512, "width": 512,
         "resolution_m": 20.0, "regional": False, "distance_m": 10_000.0, "tile_x": 192,
         "tile_y": 192, "tile_w": 128, "tile_h": 128, "azimuths": 1440, "degrees": True},
        # The benchmark's tile: site DEM plus regional DEM, 200 km rays.
        {"name": "tile-site", "kind": "tile", "height": 4096, "width": 4096,
         "resolution_m": 5.0, "regional": True, "distance_m": 200_000.0, "tile_x": 1984,
         "tile_y": 2016, "tile_w": 128, "tile_h": 128, "azimuths": 1440, "degrees": False},
        # The drop-in session on host segments, slopes back on the host: the
        # last, ragged tile column of a DEM whose sides are not whole tiles.
        {"name": "session-edge", "kind": "session", "height": 1000, "width": 1100,
         "resolution_m": 10.0, "regional": True, "distance_m": 60_000.0, "tile_x": 1024,
         "tile_y": 384, "tile_w": 76, "tile_h": 76, "azimuths": 1440},
        # The multi-site batch: uneven sites, one regional DEM, skip ladder.
        {"name": "sites-ladder", "kind": "sites", "sites": 8, "traversal": "ladder",
         "distance_m": 200_000.0, "azimuths": 1440},
        # A month of 6-hourly sun fractions of one patch (float32).
        {"name": "lightmap-month", "kind": "lightmap", "tiles": 1, "steps": 125,
         "step_hours": 6.0, "bytes": False, "valid_w": 128, "valid_h": 128},
        # A year of hourly lightmap bytes of four patches.
        {"name": "lightmap-year", "kind": "lightmap", "tiles": 4, "steps": 8761,
         "step_hours": 1.0, "bytes": True, "valid_w": 128, "valid_h": 128},
        # PSR masks of four patches over three years of hourly vectors.
        {"name": "psr", "kind": "psr", "tiles": 4, "steps": 26_281, "step_hours": 1.0,
         "valid_w": 128, "valid_h": 128},
        # Mission duration: Sun and Earth conditions over one year, 12 windows.
        {"name": "mission", "kind": "mission", "tiles": 2, "steps": 8761, "step_hours": 1.0,
         "earth": True, "windows": 12, "valid_w": 128, "valid_h": 117},
        # Writing and reading one .cbin tile.
        {"name": "codec-encode", "kind": "codec", "decode": False, "valid_w": 128,
         "valid_h": 128},
        {"name": "codec-decode", "kind": "codec", "decode": True, "valid_w": 128,
         "valid_h": 128},
        # One step of a gradient descent on terrain heights: 20 km rays of one
        # tile, a month of two-hour steps.
        {"name": "adjoint", "kind": "adjoint", "height": 1024, "width": 1024,
         "resolution_m": 10.0, "distance_m": 20_000.0, "tiles": 1, "steps": 355,
         "step_hours": 2.0},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(("tile", "tile", "session", "sites", "sites", "lightmap", "lightmap",
                       "psr", "mission", "haven", "visibility", "codec", "adjoint"))
    if kind in ("tile", "session"):
        # DEM sides from a few tiles up to the site scale, not whole tiles.
        height, width = _log_int(rng, 150, 4096), _log_int(rng, 150, 4096)
        tile_w = rng.choice((128, 128, rng.randrange(9, 129)))
        tile_h = rng.choice((tile_w, rng.randrange(1, tile_w + 1)))
        case = {"kind": kind, "height": height, "width": width,
                "resolution_m": rng.choice((5.0, 10.0, 20.0, 40.0, 118.45)),
                "regional": rng.random() < 0.5,
                "distance_m": math.exp(rng.uniform(math.log(5e3), math.log(2e5))),
                "tile_x": rng.randrange(0, max(1, width - tile_w // 2)),
                "tile_y": rng.randrange(0, max(1, height - tile_h // 2)),
                "tile_w": tile_w, "tile_h": tile_h,
                "azimuths": rng.choice((1440, 1440, 720, 360, _log_int(rng, 36, 1440)))}
        if kind == "tile":
            case["degrees"] = rng.random() < 0.5
        return case
    if kind == "sites":
        traversal = rng.choice(("ladder", "relative-ladder", "exact", "relative"))
        return {"kind": kind, "sites": rng.randrange(1, 7 if "ladder" in traversal else 3),
                "traversal": traversal,
                "distance_m": math.exp(rng.uniform(math.log(2e4), math.log(2e5))),
                "azimuths": rng.choice((1440, 720, 360))}
    if kind == "codec":
        # A ragged tile is stored whole, -50 deg outside its valid part.
        return {"kind": kind, "decode": rng.random() < 0.5, "valid_w": rng.randrange(1, 128),
                "valid_h": rng.randrange(1, 129)}
    if kind == "adjoint":
        return {"kind": kind, "height": _log_int(rng, 200, 2048),
                "width": _log_int(rng, 200, 2048),
                "resolution_m": rng.choice((5.0, 10.0, 20.0)),
                "distance_m": math.exp(rng.uniform(math.log(5e3), math.log(2e4))),
                "tiles": rng.randrange(1, 3), "steps": _log_int(rng, 24, 720),
                "step_hours": rng.choice((1.0, 2.0, 6.0))}
    case = {"kind": kind, "tiles": rng.randrange(1, 5), "steps": _log_int(rng, 31, 17_545),
            "step_hours": rng.choice((1.0, 1.0, 2.0, 6.0)),
            "valid_w": rng.choice((128, rng.randrange(1, 129))),
            "valid_h": rng.choice((128, rng.randrange(1, 129)))}
    if kind == "lightmap":
        case["bytes"] = rng.random() < 0.5
        if not case["bytes"]:
            case["steps"] = min(case["steps"], 4383)
    elif kind == "mission":
        case["earth"] = rng.random() < 0.5
        case["windows"] = rng.randrange(1, 37)
    return case


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

def _generator(seed, stream):
    generator = torch.Generator(device="cuda")
    generator.manual_seed((int(seed) * 1_000_003 + stream * 7919) % (1 << 62))
    return generator


def _numbers(seed, stream):
    return np.random.default_rng((int(seed) % (1 << 62), stream))


def _terrain(seed, stream, height, width, resolution_m, *, sigma_m=150.0, craters=None,
             crater_max_m=8000.0, tilt_m=0.0):
    """float32[height, width] heights on the GPU: fBm (Hurst 0.8) plus bowl
    craters of power-law diameters with raised rims, plus a planar tilt."""
    generator = _generator(seed, stream)
    ky = torch.fft.fftfreq(height, device="cuda", dtype=torch.float32)[:, None]
    kx = torch.fft.rfftfreq(width, device="cuda", dtype=torch.float32)[None, :]
    k = torch.sqrt(kx * kx + ky * ky)
    k[0, 0] = 1.0
    amplitude = k ** -1.8
    amplitude[0, 0] = 0.0
    noise = torch.randn((2, *k.shape), generator=generator, device="cuda")
    surface = torch.fft.irfft2(torch.complex(noise[0] * amplitude, noise[1] * amplitude),
                               s=(height, width))
    surface = (surface - surface.mean()) * (sigma_m / surface.std())
    count = max(8, height * width // 28_000) if craters is None else craters
    numbers = _numbers(seed, stream)
    inverse = 1.0 / 100.0, 1.0 / min(crater_max_m, max(200.0, 0.25 * resolution_m *
                                                       min(height, width)))
    diameters = 1.0 / (inverse[0] - numbers.uniform(size=count) * (inverse[0] - inverse[1]))
    centers = numbers.uniform(size=(count, 2)) * (width, height)
    for diameter, (cx, cy) in zip(diameters, centers):
        radius_px = 0.5 * diameter / resolution_m
        reach = max(2, math.ceil(3.0 * radius_px))
        x0, x1 = max(0, int(cx) - reach), min(width, int(cx) + reach + 1)
        y0, y1 = max(0, int(cy) - reach), min(height, int(cy) + reach + 1)
        x = torch.arange(x0, x1, device="cuda") - cx
        y = torch.arange(y0, y1, device="cuda") - cy
        r = torch.hypot(x[None, :], y[:, None]).div_(max(radius_px, 1e-6))
        surface[y0:y1, x0:x1] += torch.where(
            r < 1.0, 0.24 * diameter * r * r - 0.2 * diameter,
            0.04 * diameter / r.clamp_min(1.0) ** 3)
    if tilt_m:
        surface += torch.linspace(-0.5 * tilt_m, 0.5 * tilt_m, width, device="cuda")
    return surface.float().contiguous()


def _grid(heights, resolution_m, latitude_deg, longitude_deg):
    """DemGrid centred on a latitude / longitude, south-polar stereographic."""
    height, width = heights.shape
    latitude, longitude = math.radians(latitude_deg), math.radians(longitude_deg)
    scale = 2.0 * RADIUS_M * math.cos(latitude) / (1.0 - math.sin(latitude))
    x, y = scale * math.sin(longitude), scale * math.cos(longitude)
    transform = np.array((x - 0.5 * width * resolution_m, resolution_m, 0.0,
                          y + 0.5 * height * resolution_m, 0.0, -resolution_m))
    return DemGrid(heights.cpu().numpy(), transform, ProjectionParameters.south_polar(RADIUS_M))


def _march_grids(case, seed):
    heights = _terrain(seed, 1, case["height"], case["width"], case["resolution_m"])
    grids = [_grid(heights, case["resolution_m"], -85.0, 30.0)]
    if case.get("regional"):
        grids.append(_grid(_terrain(seed, 2, 2000, 2000, 240.0, sigma_m=1200.0, craters=0,
                                    tilt_m=2000.0), 240.0, -85.0, 30.0))
    return grids


def _session():
    session = CudaSession(0)
    session.set_stream(torch.cuda.current_stream().cuda_stream)
    return session


def _sun_vectors(hours, longitude0_deg):
    days = hours / 24.0
    latitude = np.radians(1.54) * np.sin(2.0 * np.pi * days / 346.6)
    longitude = np.radians(longitude0_deg) - 2.0 * np.pi * days / 29.53
    return AU_M * np.stack((np.cos(latitude) * np.cos(longitude),
                            np.cos(latitude) * np.sin(longitude), np.sin(latitude)), axis=1)


def _earth_vectors(hours):
    days = hours / 24.0
    latitude = np.radians(6.7) * np.sin(2.0 * np.pi * days / 27.21)
    longitude = np.radians(7.9) * np.sin(2.0 * np.pi * days / 27.55)
    return EARTH_M * np.stack((np.cos(latitude) * np.cos(longitude),
                               np.cos(latitude) * np.sin(longitude), np.sin(latitude)), axis=1)


def _vectors(case, seed):
    hours = np.arange(case["steps"]) * case["step_hours"] + 24.0 * (seed % 9973)
    return _sun_vectors(hours, 17.0 * (seed % 21)), _earth_vectors(hours)


def _horizon_tile(heights, resolution_m, tile_x, tile_y):
    """[16384, 1440] horizon elevations (deg) of a tile of `heights`: per
    pixel and azimuth the steepest of 60 terrain samples between 30 m and
    10 km, less the drop of the sphere."""
    rows, columns = heights.shape
    flat = heights.reshape(-1)
    y, x = torch.meshgrid(torch.arange(tile_y, tile_y + SIDE, device="cuda"),
                          torch.arange(tile_x, tile_x + SIDE, device="cuda"), indexing="ij")
    y, x = y.reshape(-1, 1).float(), x.reshape(-1, 1).float()
    own = flat[(y.long() * columns + x.long())]
    azimuth = torch.arange(AZIMUTHS, device="cuda") * (2.0 * math.pi / AZIMUTHS)
    east, south = torch.sin(azimuth)[None, :], -torch.cos(azimuth)[None, :]
    best = torch.full((PLANE, AZIMUTHS), -1e9, device="cuda")
    for k in range(60):
        distance = 30.0 * (10_000.0 / 30.0) ** (k / 59.0)
        px = (x + east * (distance / resolution_m)).clamp_(0, columns - 1).round_()
        py = (y + south * (distance / resolution_m)).clamp_(0, rows - 1).round_()
        rise = flat[py.mul_(columns).add_(px).long()].sub_(own)
        rise.div_(distance).sub_(distance / (2.0 * RADIUS_M))
        torch.maximum(best, rise, out=best)
    return torch.rad2deg(torch.atan(best))


def _light_inputs(case, seed):
    """(grid, patches, horizons [n, 16384, 1440], patch heights [n, 128, 128])."""
    tiles = case.get("tiles", 1)
    valid_w, valid_h = case.get("valid_w", SIDE), case.get("valid_h", SIDE)
    # The last patch is the ragged one: the DEM ends with its valid part.
    height, width = 3 * SIDE + valid_h, (tiles + 1) * SIDE + valid_w
    heights = _terrain(seed, 3, 5 * SIDE, (tiles + 2) * SIDE, 20.0)
    grid = _grid(heights[:height, :width].contiguous(), 20.0, -86.0, 30.0 + seed % 7)
    patches, horizons = [], torch.full((tiles, SIDE, SIDE, AZIMUTHS), -50.0, device="cuda")
    dems = torch.zeros((tiles, SIDE, SIDE), device="cuda")
    for i in range(tiles):
        last = i == tiles - 1
        w, h = (valid_w, valid_h) if last else (SIDE, SIDE)
        tile_x, tile_y = (i + 2) * SIDE if last else i * SIDE, 3 * SIDE if last else 2 * SIDE
        patches.append(PatchDescriptor(i, tile_x, tile_y, tile_x // SIDE, tile_y // SIDE, w, h))
        tile = _horizon_tile(heights, 20.0, tile_x, tile_y)
        horizons[i, :h, :w] = tile.view(SIDE, SIDE, AZIMUTHS)[:h, :w]
        dems[i, :h, :w] = torch.from_numpy(
            grid.elevation_m[tile_y:tile_y + h, tile_x:tile_x + w]).cuda()
    return grid, patches, horizons.view(tiles, PLANE, AZIMUTHS), dems


def _months(case):
    """A month band (30.44 days) per step."""
    return (np.arange(case["steps"]) * case["step_hours"] / (24.0 * 30.44)).astype(np.int32)


def _windows(case):
    """Equal candidate start windows over the time axis."""
    edges = np.linspace(0, case["steps"], case["windows"] + 1).astype(np.int32)
    return np.stack((edges[:-1], edges[1:]), axis=1)


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind == "tile":
        session = state["session"] = _session()
        grids = _march_grids(case, seed)
        state["dems"] = [session.upload_dem_grid(g) for g in grids]
        centers = (case["tile_w"] // SUBPATCH + 2) ** 2
        state["centers"] = centers
        state["segments"] = torch.empty(case["azimuths"] * centers * len(grids) * 18,
                                        device="cuda")
        state["out"] = torch.empty((case["tile_w"] * case["tile_h"], case["azimuths"]),
                                   device="cuda")
    elif kind == "session":
        session = state["session"] = _session()
        grids = _march_grids(case, seed)
        state["pyramids"] = [session.build_max_pyramid(g) for g in grids]
        dems = [session.upload_dem_grid(g) for g in grids]
        state["segments"] = session.generate_segments(
            dems, tile_column=case["tile_x"], tile_row=case["tile_y"],
            tile_width=case["tile_w"], azimuth_count=case["azimuths"],
            maximum_distance_m=case["distance_m"], observer_elevation_m=2.0,
            subpatch_size=SUBPATCH)
        for dem in dems:
            dem.close()
    elif kind == "sites":
        session = state["session"] = _session()
        numbers = _numbers(seed, 4)
        regional = session.upload_dem_grid(
            _grid(_terrain(seed, 2, 2000, 2000, 240.0, sigma_m=1200.0, craters=0,
                           tilt_m=2000.0), 240.0, -90.0, 0.0))
        tiles = []
        for i in range(case["sites"]):
            size = int(round(math.exp(numbers.uniform(math.log(256), math.log(2048)))))
            resolution = float(numbers.choice((5.0, 10.0, 20.0, 40.0)))
            grid = _grid(_terrain(seed, 10 + i, size, size, resolution), resolution,
                         float(numbers.uniform(-89.5, -83.0)),
                         float(numbers.uniform(0.0, 360.0)))
            tiles.append(SiteTile((session.upload_dem_grid(grid), regional),
                                  (size - SIDE) // 2, (size - SIDE) // 2,
                                  case["distance_m"], 2.0))
        state["tiles"] = tiles
        state["out"] = torch.empty((case["sites"], PLANE, case["azimuths"]), device="cuda")
    elif kind == "codec":
        _, _, horizons, _ = _light_inputs(case, seed)
        state["codec"] = TileCodec()
        if case["decode"]:
            state["payload"] = state["codec"].encode(horizons[0].cpu().numpy())
        else:
            state["degrees"] = horizons[0].contiguous()
            state["payload"] = torch.zeros(MAX_PAYLOAD_BYTES, dtype=torch.uint8, device="cuda")
    elif kind == "adjoint":
        from lunarscout_b200.adjoint import SunLossProblem

        session = state["session"] = _session()
        heights = _terrain(seed, 1, case["height"], case["width"], case["resolution_m"])
        grid = _grid(heights, case["resolution_m"], -85.0, 30.0)
        numbers = _numbers(seed, 5)
        tiles = [(max(0, (case["width"] - case["tiles"] * SIDE) // 2) + i * SIDE,
                  (case["height"] - SIDE) // 2) for i in range(case["tiles"])]
        weights = numbers.uniform(size=(case["tiles"], SIDE, SIDE)).astype(np.float32)
        weights[numbers.uniform(size=weights.shape) < 0.3] = 0.0
        state["problem"] = SunLossProblem(session, [grid], tiles, weights,
                                          _vectors(case, seed)[0],
                                          maximum_distance_m=case["distance_m"],
                                          observer_elevation_m=2.0)
        state["heights"] = [heights]
    else:
        grid, patches, horizons, dems = _light_inputs(case, seed)
        count = len(patches)
        chain = state["chain"] = ProductChain([grid])
        state["batch"] = PatchBatch(
            patches, horizons, dems, np.repeat(grid.geo_transform[None], count, 0),
            np.repeat(grid.projection.as_array()[None], count, 0),
            np.array([(p.tile_x, p.tile_y, p.width, p.height) for p in patches], np.int32))
        state["sun"], state["earth"] = _vectors(case, seed)
        state["hours"] = np.full(case["steps"], case["step_hours"])
        if kind == "mission":
            state["windows"] = _windows(case)
        if kind == "haven":
            state["months"] = _months(case)
    torch.cuda.synchronize()
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "tile":
        session = state["session"]
        session.generate_segments_device(
            state["dems"], state["segments"].data_ptr(), tile_column=case["tile_x"],
            tile_row=case["tile_y"], tile_width=case["tile_w"],
            azimuth_count=case["azimuths"], maximum_distance_m=case["distance_m"],
            observer_elevation_m=2.0, subpatch_size=SUBPATCH)
        session.march_all_passes_device(
            state["segments"].data_ptr(), case["azimuths"], state["centers"], state["dems"],
            tile_column=case["tile_x"], tile_row=case["tile_y"], tile_width=case["tile_w"],
            tile_height=case["tile_h"], subpatch_size=SUBPATCH, observer_elevation_m=2.0,
            device_out=state["out"].data_ptr(), degrees=case["degrees"])
        return state["out"]
    if kind == "session":
        return state["session"].subpatch_hierarchical_all_passes(
            state["segments"], state["pyramids"], tile_column=case["tile_x"],
            tile_row=case["tile_y"], tile_width=case["tile_w"], tile_height=case["tile_h"],
            subpatch_size=SUBPATCH, observer_elevation_m=2.0)[0]
    if kind == "sites":
        state["session"].march_sites(
            state["tiles"], device_out=state["out"].data_ptr(),
            azimuth_count=case["azimuths"], subpatch_size=SUBPATCH,
            traversal=case["traversal"], degrees=True)
        return state["out"]
    if kind == "codec":
        if case["decode"]:
            return state["codec"].decode(state["payload"])
        size = state["codec"].encode_device(state["degrees"].data_ptr(),
                                            state["payload"].data_ptr())
        return size, state["payload"]
    if kind == "adjoint":
        loss = state["problem"].forward_value(state["heights"])
        return loss, state["problem"].backward_value()
    chain, batch = state["chain"], state["batch"]
    if kind == "lightmap":
        if case["bytes"]:
            return chain.sun_fraction_bytes(batch, state["sun"])
        return chain.sun_fractions(batch, state["sun"])
    if kind == "psr":
        return chain.psr(batch, state["sun"])
    if kind == "mission":
        return chain.mission_durations(
            batch, state["sun"], sample_hours=state["hours"], start_windows=state["windows"],
            earth_vectors_m=state["earth"] if case["earth"] else None)
    if kind == "haven":
        return chain.safe_haven(batch, state["sun"], state["earth"],
                                month_index_of=state["months"],
                                band_count=int(state["months"][-1]) + 1,
                                time_step_hours=case["step_hours"])
    return chain.earth_visibility(batch, state["earth"])


# ---------------------------------------------------------------------------
# work / exact
# ---------------------------------------------------------------------------

def _march_work(rays, azimuths, resolution_m, distance_m, extent_m, regional, ladder,
                cells, pixels_w):
    """Bytes: DEM cells and segments read once, slopes written once.  Flops:
    a footprint-limited ray takes about 1 / ln(1 + 0.25 deg) steps per factor
    of e in distance from the first kilometre on, two samples per pixel of
    path before it (67 + 31 flops a step with its node visit, 66 a sample);
    the ladder takes about a twelfth of those steps."""
    near = 2.0 * min(1000.0, distance_m) / resolution_m
    reach = distance_m if regional else min(distance_m, 0.6 * extent_m)
    far = 229.0 * math.log(max(1.0, reach / 1000.0)) * (1.0 / 12.0 if ladder else 1.0)
    centers = (pixels_w // SUBPATCH + 2) ** 2
    passes = 2 if regional else 1
    return {"bytes": 4.0 * (cells + rays + azimuths * centers * 18 * passes),
            "flops": rays * (98.0 * far + 164.0 * near)}


def work(case):
    kind = case["kind"]
    if kind in ("tile", "session"):
        rays = case["tile_w"] * case["tile_h"] * case["azimuths"]
        cells = case["height"] * case["width"] + (4_000_000 if case["regional"] else 0)
        extent = case["resolution_m"] * min(case["height"], case["width"])
        return _march_work(rays, case["azimuths"], case["resolution_m"], case["distance_m"],
                           extent, case["regional"], False, cells, case["tile_w"])
    if kind == "sites":
        one = _march_work(PLANE * case["azimuths"], case["azimuths"], 14.0, case["distance_m"],
                          10_000.0, True, "ladder" in case["traversal"], 600_000, SIDE)
        return {key: case["sites"] * value for key, value in one.items()}
    if kind == "codec":
        return {"bytes": PLANE * AZIMUTHS * 5.2, "flops": PLANE * AZIMUTHS * 6.0}
    if kind == "adjoint":
        tile = _march_work(PLANE * AZIMUTHS, AZIMUTHS, case["resolution_m"],
                           case["distance_m"],
                           case["resolution_m"] * min(case["height"], case["width"]),
                           False, True, 0, SIDE)
        cells = case["height"] * case["width"]
        samples = PLANE * case["steps"]
        return {"bytes": case["tiles"] * tile["bytes"] + 12.0 * cells,
                "flops": case["tiles"] * (tile["flops"] + 2 * 60.0 * samples)}
    pixels = (case["tiles"] - 1) * PLANE + case["valid_w"] * case["valid_h"]
    samples = pixels * case["steps"]
    horizons = 4.0 * pixels * AZIMUTHS
    if kind == "lightmap":
        out = case["tiles"] * PLANE * case["steps"] * (1.0 if case["bytes"] else 4.0)
        return {"bytes": horizons + out, "flops": 150.0 * samples}
    if kind == "psr":
        # At most 5 x 1440 of the vectors are kept; most pixels see the Sun in
        # the first few of them.
        return {"bytes": horizons + 24.0 * case["steps"],
                "flops": 200.0 * 5 * case["steps"] + 40.0 * pixels * min(case["steps"], 200)}
    both = 2 if kind == "haven" or case.get("earth") else 1
    planes = {"mission": case.get("windows", 1), "haven": int(_months(case)[-1]) + 1,
              "visibility": 1}[kind]
    per_sample = 50.0 if kind == "visibility" else 150.0 + (50.0 if both == 2 else 0.0)
    return {"bytes": horizons + 4.0 * pixels * planes, "flops": per_sample * samples}


def _frames(case, grid, patches, dems):
    """Per patch: float64 rotation rows (east, north, up) and translation of
    every pixel, [16384, 3, 4]."""
    out = []
    for patch, heights in zip(patches, dems):
        rows, columns = torch.meshgrid(torch.arange(SIDE, device="cuda", dtype=torch.float64),
                                       torch.arange(SIDE, device="cuda", dtype=torch.float64),
                                       indexing="ij")
        gt = grid.geo_transform
        x = (gt[0] + gt[1] * (columns + patch.tile_x)).reshape(-1)
        y = (gt[3] + gt[5] * (rows + patch.tile_y)).reshape(-1)
        angle = 2.0 * torch.atan(torch.hypot(x, y) / (2.0 * RADIUS_M))
        latitude, longitude = angle - 0.5 * math.pi, torch.atan2(x, y)
        radius = RADIUS_M + heights.reshape(-1).double()
        sin_lat, cos_lat = torch.sin(latitude), torch.cos(latitude)
        sin_lon, cos_lon = torch.sin(longitude), torch.cos(longitude)
        zero = torch.zeros_like(radius)
        out.append(torch.stack((
            torch.stack((-sin_lon, cos_lon, zero, zero), 1),
            torch.stack((-sin_lat * cos_lon, -sin_lat * sin_lon, cos_lat, zero), 1),
            torch.stack((cos_lat * cos_lon, cos_lat * sin_lon, sin_lat, -radius), 1)), 1))
    return out


def _directions(frame, vectors):
    """(azimuth, elevation) in degrees of `vectors` [t, 3] at every pixel."""
    homogeneous = torch.cat((vectors, torch.ones_like(vectors[:, :1])), 1)
    local = torch.einsum("pij,tj->itp", frame, homogeneous)
    azimuth = torch.rad2deg(torch.atan2(local[0], local[1])) % 360.0
    return azimuth, torch.rad2deg(torch.atan2(local[2], torch.hypot(local[0], local[1])))


def _fraction(horizons, azimuth, elevation):
    """Visible fraction of a 0.27-deg disk in 16 columns against the
    interpolated horizon; horizons float64 [16384, 1440]."""
    position = (azimuth - 0.395) * 4.0
    left = torch.trunc(position)
    offset = position - left
    total, photons = 0.0, torch.zeros_like(azimuth)
    for k in range(16):
        half = math.sqrt(64.0 - (7.5 - k) ** 2) / 8.0 * 0.27
        place = offset + 0.135 * k
        cell = torch.floor(place.clamp_min(0.0))
        index = (left + cell).long() % AZIMUTHS
        h0 = torch.gather(horizons, 1, index.t()).t()
        h1 = torch.gather(horizons, 1, ((index + 1) % AZIMUTHS).t()).t()
        h = h0 + (place - cell) * (h1 - h0)
        photons += (elevation + half - h).clamp(0.0, 2.0 * half)
        total += 2.0 * half
    return photons / total


def _margin(horizons, azimuth, elevation):
    position = azimuth * 4.0
    left = torch.floor(position)
    index = left.long() % AZIMUTHS
    h0 = torch.gather(horizons, 1, index.t()).t()
    h1 = torch.gather(horizons, 1, ((index + 1) % AZIMUTHS).t()).t()
    return elevation - (h0 + (position - left) * (h1 - h0))


def _signal(frame, horizons, vectors, signal, block=256):
    """[T, 16384] of a signal function, evaluated in blocks of steps."""
    table = torch.from_numpy(vectors).cuda()
    return torch.cat([signal(horizons, *_directions(frame, table[t:t + block]))
                      for t in range(0, len(table), block)])


def _longest_runs(case, on, windows):
    """Longest run of true samples per start window, [I, 16384] hours."""
    first = torch.from_numpy(windows[:, :1].astype(np.int64)).cuda()
    end = torch.from_numpy(windows[:, 1:].astype(np.int64)).cuda()
    start = torch.full((1, PLANE), -1, dtype=torch.int64, device="cuda")
    best = torch.zeros((len(windows), PLANE), dtype=torch.int64, device="cuda")
    for t in range(len(on)):
        start = torch.where(on[t], torch.where(start < 0, t, start), -1)
        begin = torch.maximum(start, first)
        live = on[t] & (begin < end) & (begin <= t)
        best = torch.maximum(best, torch.where(live, t + 1 - begin, 0))
    return best.double() * case["step_hours"]


def _haven(case, low, outage, months):
    """Longest low-Sun run that met an outage in each band, [bands, 16384]."""
    length = torch.zeros(low.shape, dtype=torch.int32, device="cuda")
    length[0] = low[0]
    for t in range(1, len(low)):
        length[t] = torch.where(low[t], length[t - 1] + 1, 0)
    for t in range(len(low) - 2, -1, -1):
        length[t] = torch.where(low[t] & low[t + 1], length[t + 1], length[t])
    out = []
    for band in range(int(months[-1]) + 1):
        steps = slice(int(np.searchsorted(months, band)), int(np.searchsorted(months, band + 1)))
        hit = torch.where(low[steps] & outage[steps], length[steps], 0).amax(0)
        both = outage[steps].any(0) & (~outage[steps]).any(0)
        out.append(torch.where(both, hit.double() * case["step_hours"], math.nan))
    return torch.stack(out)


def exact(case, seed):
    kind = case["kind"]
    # The march has no value that is independent of its step decisions short
    # of a restatement of the march (far above the time allowed on the host);
    # PSR masks, lightmap bytes and encoded tiles are whole numbers.
    if kind in ("tile", "session", "sites", "adjoint", "psr"):
        return None
    if kind == "codec":
        if not case["decode"]:
            return None
        _, _, horizons, _ = _light_inputs(case, seed)
        # What the format stores: samples quantised by float32(32767 / 50),
        # differences limited to 15 bits, read back in steps of 50 / 32767.
        scaled = horizons[0].clamp(-50.0, 50.0) * float(np.float32(32767.0) / np.float32(50.0))
        scaled = scaled.double()
        q = torch.where(scaled >= 0, torch.floor(scaled + 0.5), torch.ceil(scaled - 0.5))
        for k in range(1, AZIMUTHS):
            q[:, k] = q[:, k - 1] + (q[:, k] - q[:, k - 1]).clamp(-16384, 16383)
        return (q * (50.0 / 32767.0)).cpu().numpy()
    if kind == "lightmap" and (case["bytes"] or case["tiles"] * case["steps"] > 5000):
        return None
    if kind in ("mission", "haven") and case["tiles"] * case["steps"] > 20_000:
        return None
    grid, patches, horizons, dems = _light_inputs(case, seed)
    sun, earth = _vectors(case, seed)
    out = []
    for patch, frame, rows in zip(patches, _frames(case, grid, patches, dems), horizons):
        rows = rows.double()
        if kind == "lightmap":
            full = _signal(frame, rows, sun, _fraction)
            valid = torch.zeros((SIDE, SIDE), device="cuda", dtype=torch.bool)
            valid[:patch.height, :patch.width] = True
            out.append(torch.where(valid.view(-1), full, 0.0))
            continue
        if kind == "visibility":
            planes = (_signal(frame, rows, earth, _margin) >= 0.0).double().mean(0)[None]
        elif kind == "mission":
            on = _signal(frame, rows, sun, _fraction) >= 0.5
            if case["earth"]:
                on &= _signal(frame, rows, earth, _margin) >= 0.0
            planes = _longest_runs(case, on, _windows(case))
        else:
            planes = _haven(case, _signal(frame, rows, sun, _fraction) < 0.2,
                            _signal(frame, rows, earth, _margin) < 2.0, _months(case))
        planes = planes.view(-1, SIDE, SIDE)[:, :patch.height, :patch.width].cpu().numpy()
        out.append(np.ascontiguousarray(planes[0] if kind == "visibility" else planes))
    return torch.stack(out) if kind == "lightmap" else out
