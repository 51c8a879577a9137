"""Damaged rows in run-length .hdr files large enough for the device's row walk: packet counts of zero, counts
beyond the end of a row, and a row that is not run-length.  The oracle's parser decides what is a file."""
import numpy as np
import pytest

import oracle_binding as ob
from test_gpu_film_io import ctx, torch_cuda  # noqa: F401
from test_gpu_hdr_rows import _check, _file, _row

pytestmark = pytest.mark.gpu

W, H, AT = 700, 270, 41


@pytest.mark.parametrize("at", [0, AT, H - 1])
@pytest.mark.parametrize("what", ["zero_first", "zero_last", "zeros", "long_run", "long_dump"])
def test_bad_packet_counts(ctx, oracle, torch_cuda, tmp_path, what, at):  # noqa: F811
    parts = _file(W, H, 5, 0.1)
    row = parts[1 + at]
    if what == "zero_first":  # the first packet's count
        row = row[:4] + bytes([0]) + row[5:]
    elif what == "zero_last":  # after all of a plane but its last value, so the walk meets the zero late
        row = row[:4] + bytes([128 + 127, 9]) * 5 + bytes([128 + 64, 9, 0, 9]) + row[4:]
    elif what == "zeros":
        row = row[:4] + bytes(len(row) - 4)
    elif what == "long_run":  # 635 values, then 100 more than the row has
        row = row[:4] + bytes([128 + 127, 9]) * 5 + bytes([128 + 100, 9]) + row[4:]
    else:
        row = row[:4] + bytes([128 + 127, 9]) * 5 + bytes([100]) + bytes(100) + row[4:]
    parts[1 + at] = row
    data = b"".join(parts)
    assert ob.hdr_parse(data)[0] != 0
    _check(ctx, torch_cuda, tmp_path / "f.hdr", data)


@pytest.mark.parametrize("at", [1, AT, H - 1])
def test_row_that_is_not_run_length(ctx, oracle, torch_cuda, tmp_path, at):  # noqa: F811
    parts = _file(W, H, 5, 0.1)
    parts[1 + at] = bytes([1, 2, 3, 4]) * W
    _check(ctx, torch_cuda, tmp_path / "f.hdr", b"".join(parts))


def test_one_changed_byte_at_a_time(ctx, oracle, torch_cuda, tmp_path):  # noqa: F811
    """Every byte of one row's header and first packets, set to values that a walk treats differently."""
    rng = np.random.default_rng(8)
    parts = _file(W, H, 6, 0.1)
    row = _row(rng, W, 0.0, 0.5)
    for k in range(24):
        for value in (0, 2, 128, 129, 255):
            parts[1 + AT] = row[:k] + bytes([value]) + row[k + 1:]
            _check(ctx, torch_cuda, tmp_path / "f.hdr", b"".join(parts))
