"""Rows with jumps beyond 15 bits, whose clamped differences carry into the
samples after them: noise, jumps at every place of the 32-sample groups, runs of
clamped samples across groups, alternating extremes and infinities.  Bytes must
equal the CPU oracle's."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import products

pytestmark = pytest.mark.gpu

AZ = 1440


def _rows():
    rng = np.random.default_rng(33)
    rows = [rng.uniform(-50.0, 50.0, AZ) for _ in range(6)]
    rows += [rng.choice((-50.0, 50.0), AZ), np.where(np.arange(AZ) % 2, 50.0, -50.0),
             rng.choice((-np.inf, 3.0, 49.0), AZ), np.linspace(-50.0, 50.0, AZ)]
    for place in (1, 29, 30, 31, 32, 33, 63, 64, 1437, 1438, 1439):
        row = rng.uniform(-1.0, 1.0, AZ) - 48.0
        row[place:] += 96.0
        rows.append(row)
        spike = rng.uniform(-1.0, 1.0, AZ)
        spike[place] = -np.inf
        rows.append(spike)
    for width in (2, 3, 4, 5, 40):
        row = np.full(AZ, 45.0)
        for start in range(28, AZ, 97):
            row[start:start + width] = -50.0
        rows.append(row)
    # 25 degrees are 16383.5 steps: differences around the clamp's own edge.
    rows.append(np.where(np.arange(AZ) % 2, 12.5, -12.5) + rng.uniform(-2e-3, 2e-3, AZ))
    return np.stack(rows).astype(np.float32)


def test_clamped_rows_encode_as_the_oracle():
    from lunarscout_b200.file_format import TileCodec

    rows = _rows()
    degrees = np.zeros((16384, AZ), np.float32)
    degrees[:len(rows)] = rows
    codec = TileCodec()
    try:
        payload = codec.encode(degrees)
        head = b"".join(products.encode_tile(row[None]) for row in rows)
        assert payload[:len(head)] == head
        decoded = codec.decode(payload)[:len(rows)]
    finally:
        codec.close()
    zero = products.encode_tile(degrees[-1:])
    assert payload[len(head):] == zero * (16384 - len(rows))
    expected = products.decode_tile(payload)[:len(rows)]
    np.testing.assert_array_equal(decoded, expected)
