"""Run-length .hdr files large enough (320 KB, or a megapixel) that the device finds and expands their rows: against the oracle's parser,
with packets of every length, a row header's bytes inside packet data, damaged and cut files, and files
that stop being run-length.  Whole numbers and exact scalings throughout: the bits are equal."""
import numpy as np
import pytest

import oracle_binding as ob
from test_film_io import header
from test_gpu_film_io import ctx, torch_cuda  # noqa: F401

pytestmark = pytest.mark.gpu


def _row(rng, w, plant, runs):
    """One row's packets over random values: dumps and runs of random lengths, and sometimes the row header
    as dump data."""
    out = bytearray([2, 2, w >> 8, w & 255])
    for _ in range(4):
        x = 0
        while x < w:
            n = int(min(w - x, rng.choice([1, 2, 3, 4, 5, 31, 32, 33, 126, 127, 128])))
            if rng.random() < runs:
                n = min(n, 127)
                out += bytes([128 + n, int(rng.integers(0, 256))])
            else:
                data = bytearray(rng.integers(0, 256, n, dtype=np.uint8).tobytes())
                if n >= 4 and rng.random() < plant:
                    data[-4:] = bytes([2, 2, w >> 8, w & 255])
                out += bytes([n]) + data
            x += n
    return bytes(out)


def _file(w, h, seed, plant=0.0, runs=0.4):
    rng = np.random.default_rng(seed)
    return [header(w, h)] + [_row(rng, w, plant, runs) for _ in range(h)]


def _check(ctx, torch, path, data):
    from axomae_b200 import native
    path.write_bytes(data)
    code, w, h, q = ob.hdr_parse(data)
    wi, hi = native.hdr_info(str(path))
    assert len(data) - 100 > 5 << 16 or (len(data) > 1 << 16 and wi * hi >= 1 << 20)
    host = np.full((hi, wi, 4), -1.0, np.float32)
    dev = torch.full((hi, wi, 4), -1.0, device="cuda")
    if code:
        with pytest.raises(native.NovaError) as e:
            ctx.hdr_read(str(path), rgba_host=host, rgba_device_ptr=dev.data_ptr())
        assert e.value.status == 15 and (host == -1.0).all()
        return
    want = ob.rgbe_decode(q.reshape(-1, 4)).reshape(h, w, 4)
    ctx.hdr_read(str(path), rgba_host=host, rgba_device_ptr=dev.data_ptr())
    assert np.array_equal(host.view(np.uint32), want.view(np.uint32))
    assert np.array_equal(dev.cpu().numpy().view(np.uint32), want.view(np.uint32))
    only = np.zeros_like(host)
    ctx.hdr_read(str(path), rgba_host=only)
    assert np.array_equal(only.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("w,h,plant,runs", [(8, 12000, 0.0, 0.4), (8, 12000, 0.3, 0.2), (257, 400, 0.0, 0.0),
                                            (514, 400, 0.2, 0.5), (1026, 1, 0.0, 0.0), (5000, 300, 0.02, 0.9),
                                            (20000, 8, 0.0, 0.1), (32767, 8, 0.01, 0.4), (300, 1100, 1.0, 0.1),
                                            (1024, 512, 0.0, 0.4), (2048, 512, 0.0, 1.0)])
def test_packets_of_every_length(ctx, oracle, torch_cuda, tmp_path, w, h, plant, runs):  # noqa: F811
    if (w, h) == (1026, 1):
        data = b"".join(_file(w, h, 1, plant, runs)) + bytes(330000)  # one row, then bytes nobody reads
    else:
        data = b"".join(_file(w, h, w + h, plant, runs))
    _check(ctx, torch_cuda, tmp_path / "f.hdr", data)


@pytest.mark.parametrize("what", ["cut", "cut_in_header", "no_last_row", "bad_count", "short_row", "flat_later", "longer"])
def test_damaged_files(ctx, oracle, torch_cuda, tmp_path, what):  # noqa: F811
    parts = _file(700, 270, 5, 0.1)
    if what == "cut":
        data = b"".join(parts)[:-40]
    elif what == "cut_in_header":
        data = b"".join(parts[:-1]) + parts[-1][:3]
    elif what == "no_last_row":
        data = b"".join(parts[:-1])
    elif what == "bad_count":
        parts[41] = parts[41][:4] + b"\\0" + parts[41][5:]
        data = b"".join(parts)
    elif what == "short_row":
        parts[41] = parts[41][:-3]
        data = b"".join(parts)
    elif what == "flat_later":
        parts[41] = b"\\1\\2\\3\\4" * 700
        data = b"".join(parts)
    else:
        data = b"".join(parts) + parts[1] + parts[2]
    _check(ctx, torch_cuda, tmp_path / "f.hdr", data)
