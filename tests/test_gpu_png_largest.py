"""The device PNG writer at the largest file it accepts: the slices that
follow the first one are then 64^3."""
import zlib

import numpy as np
import pytest

import zigtrace_b200 as zt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height", [(21846, 32764)])
def test_checksums_of_the_largest_file(width, height):
    import torch
    size = zt.png_size(width, height)
    assert (size + 31 + 8191) // 8192 - 1 == 262144
    torch.manual_seed(3)
    rgb = torch.randint(0, 256, (height, width * 3), dtype=torch.uint8, device="cuda")
    out = torch.zeros(size, dtype=torch.uint8, device="cuda")
    zt.encode_png_device(rgb.data_ptr(), width, height, out.data_ptr(), size)
    torch.cuda.synchronize()
    png = out.cpu().numpy()
    chunk = png[37:size - 16]  # the type and the data
    assert int.from_bytes(png[size - 16:size - 12].tobytes(), "big") == zlib.crc32(chunk)
    adler = 1
    host = rgb.cpu().numpy()
    for y0 in range(0, height, 4096):
        rows = host[y0:y0 + 4096]
        adler = zlib.adler32(np.concatenate([np.zeros((len(rows), 1), np.uint8), rows], axis=1).reshape(-1), adler)
    assert int.from_bytes(png[size - 20:size - 16].tobytes(), "big") == adler
