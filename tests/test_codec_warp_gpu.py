"""The warp-per-pixel .cbin codec where its grouping can go wrong, against the
CPU oracle: runs of two-byte deltas whose second bytes also have the top bit
set, crossing the 32-byte groups at every phase; one- and two-byte deltas
mixed; clamped jumps next to ordinary rows; record offsets of every alignment;
and blocks whose last delta is cut short."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import products

pytestmark = pytest.mark.gpu

AZ = 1440
STEP = np.float32(50.0) / np.float32(32767.0)


def _row(deltas):
    """Degrees whose quantised differences are `deltas` (folded into +-30000)."""
    values = np.cumsum(np.asarray(deltas, dtype=np.int64))
    folded = np.abs((values + 30000) % 120000 - 60000) - 30000
    return (folded * (50.0 / 32767.0)).astype(np.float32)


def _rows():
    rng = np.random.default_rng(21)
    rows = [_row(np.full(AZ, 0x0FF)),                      # second byte 0xff
            _row(np.where(np.arange(AZ) % 2, -0x81, 0x85))]  # alternating signs
    for phase in range(8):
        deltas = rng.integers(-60, 60, size=AZ)
        wide = (np.arange(AZ) + phase) % (3 + phase) < 2 + phase // 2
        deltas[wide] = rng.choice((200, 255, -129, -200, 63, -65, 64), size=int(wide.sum()))
        rows.append(_row(deltas))
    for edge in (62, 63, -64, -65):
        rows.append(_row(np.where(np.arange(AZ) % 2, edge, -edge)))
    jumps = _row(rng.integers(-50, 50, size=AZ))
    jumps[100::331] = 49.9
    jumps[101::331] = -49.9
    rows.append(jumps)
    rows.append(np.zeros(AZ, np.float32))
    return np.stack(rows)


@pytest.fixture(scope="module")
def codec():
    from lunarscout_b200.file_format import TileCodec

    codec = TileCodec()
    yield codec
    codec.close()


def test_special_rows_encode_and_decode_as_the_oracle(codec):
    rows = _rows()
    degrees = np.zeros((16384, AZ), np.float32)
    degrees[:len(rows)] = rows
    payload = codec.encode(degrees)
    head = products.encode_tile(rows)
    assert payload[:len(head)] == head
    blocks = payload[len(head):]
    zero = products.encode_tile(degrees[-1:])
    assert blocks == zero * (16384 - len(rows))
    expected = products.decode_tile(head + zero * (16384 - len(rows)))[:len(rows)]
    np.testing.assert_array_equal(codec.decode(payload)[:len(rows)], expected)


@pytest.mark.parametrize("row", [0, 1, 5, 13])
def test_a_cut_delta_is_refused(codec, row):
    block = products.encode_tile(_rows()[row:row + 1])
    zero = products.encode_tile(np.zeros((1, AZ), np.float32))
    for cut in (1, 2, 33):
        short = block[2:-cut]
        record = len(short).to_bytes(2, "little") + short
        with pytest.raises(ValueError):
            codec.decode(record + zero * 16383)
