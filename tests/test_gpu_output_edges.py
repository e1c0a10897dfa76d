"""The device output stage at its edges: the encode's single-precision
estimate beside every rounding boundary, special values, options outside the
estimate's range, odd counts and unaligned buffers; the PNG at sizes around
its segments and slices, with image and file at any alignment."""
import numpy as np
import pytest

import zigtrace_b200 as zt

pytestmark = pytest.mark.gpu


def _mapped(x, tonemap):
    if tonemap == "reinhard":
        return x / (1.0 + x)
    if tonemap == "aces":
        return (x * (2.51 * x + 0.03)) / (x * (2.43 * x + 0.59) + 0.14)
    return x


def _reference(v, tonemap, gamma, exposure):
    """Output.encode (image.zig:14-37) in f64: c * 255."""
    with np.errstate(all="ignore"):
        x = np.fmax(np.where(np.isnan(v), 0.0, v) * exposure, 0.0)
        m = _mapped(x, tonemap)
        m = np.where(np.isnan(m), 1.0, np.clip(m, 0.0, 1.0))
        c = m ** (1.0 / gamma)
        return np.where(np.isnan(c), 1.0, np.clip(c, 0.0, 1.0)) * 255.0


def _boundary_inputs(tonemap, gamma, exposure):
    """Inputs whose encode lies at, and within 1e-12 .. 1e-3 of, k + 1/2."""
    grid = np.concatenate([[0.0], np.geomspace(1e-6, 1e3, 200_001)])
    m = np.clip(_mapped(grid, tonemap), 0, 1)
    k = (np.arange(255) + 0.5) / 255.0
    x = np.interp(k ** gamma, m, grid)
    eps = np.array([0.0, 1e-12, 1e-9, 1e-8, 1e-7, 1e-6, 1e-5, 1e-4, 1e-3])
    return np.concatenate([(x[:, None] * (1 + np.concatenate([eps, -eps]))).ravel()]) / exposure


SPECIAL = np.array([0.0, -0.0, np.nan, np.inf, -np.inf, -1.0, 1.0, 5e-324, 1e-310, 1e-45, 1e-38, 1e-30, 1e-29, 1e-12,
                    1e14, 1e15, 1e16, 1e38, 1e39, 1e300, -1e300])


@pytest.mark.parametrize("gamma,exposure", [(2.2, 1.0), (1.0, 0.37), (0.26, 2.0), (9.5, 1.0), (40.0, 1.0), (-1.5, 1.0),
                                            (2.2, -1.0), (2.4, 1e11)])
@pytest.mark.parametrize("tonemap", ["none", "reinhard", "aces"])
def test_encode_beside_rounding_boundaries(tonemap, gamma, exposure):
    import torch
    rng = np.random.default_rng(1)
    v = np.concatenate([SPECIAL, rng.uniform(0, 4, 50_000), 10.0 ** rng.uniform(-40, 20, 20_000),
                        _boundary_inputs(tonemap, abs(gamma), abs(exposure)) if 0.1 <= abs(1 / gamma) <= 4 else []])
    v = v[:len(v) // 3 * 3]
    d = torch.from_numpy(v).cuda()
    out = torch.empty(len(v), dtype=torch.uint8, device="cuda")
    zt.image_to_rgb8_device(d.data_ptr(), len(v) // 3, out.data_ptr(), zt.Output(tonemap, gamma, exposure))
    got = out.cpu().numpy().astype(int)
    want = _reference(v, tonemap, gamma, exposure)
    byte = np.floor(want + 0.5)
    # where two f64 pow()s may round to opposite sides (1e-12 covers both)
    sure = np.abs(want + 0.5 - np.round(want + 0.5)) > 1e-12 * 255
    assert (got[sure] == byte[sure]).all()
    assert (np.abs(got - byte) <= 1).all()


@pytest.mark.parametrize("offset", [(0, 0), (0, 1), (8, 0), (8, 3)])
@pytest.mark.parametrize("pixels", [1, 2, 3, 170, 171, 341, 342, 683])
def test_encode_counts_and_alignment(pixels, offset):
    import torch
    rng = np.random.default_rng(pixels)
    v = rng.uniform(0, 1.2, 3 * pixels)
    d = torch.zeros(3 * pixels + 1, dtype=torch.float64, device="cuda")
    d[offset[0] // 8:offset[0] // 8 + len(v)] = torch.from_numpy(v).cuda()
    out = torch.full((3 * pixels + 8,), 77, dtype=torch.uint8, device="cuda")
    zt.image_to_rgb8_device(d.data_ptr() + offset[0], pixels, out.data_ptr() + offset[1], zt.Output())
    got = out.cpu().numpy()
    want = zt.Image(pixels, 1, v.reshape(-1, 3)).to_rgb8()
    assert (got[offset[1]:offset[1] + 3 * pixels] == want).all()
    assert (got[:offset[1]] == 77).all() and (got[offset[1] + 3 * pixels:] == 77).all()


@pytest.mark.parametrize("offset", [(0, 0), (1, 0), (2, 5), (3, 31), (0, 16)])
@pytest.mark.parametrize("w,h", [(1, 1), (2, 3), (10, 1), (11, 2), (43, 61), (107, 25), (2720, 1), (2721, 1),
                                 (21845, 1), (21846, 2), (300, 219)])
def test_png_sizes_and_alignment(w, h, offset):
    import torch
    rng = np.random.default_rng(w + h)
    rgb = rng.integers(0, 256, 3 * w * h).astype(np.uint8)
    want = np.frombuffer(zt.encode_png(rgb, w, h), np.uint8)
    d = torch.zeros(3 * w * h + 4, dtype=torch.uint8, device="cuda")
    d[offset[0]:offset[0] + len(rgb)] = torch.from_numpy(rgb).cuda()
    out = torch.full((len(want) + 64,), 77, dtype=torch.uint8, device="cuda")
    zt.encode_png_device(d.data_ptr() + offset[0], w, h, out.data_ptr() + offset[1], len(want))
    got = out.cpu().numpy()
    assert (got[offset[1]:offset[1] + len(want)] == want).all()
    assert (got[:offset[1]] == 77).all() and (got[offset[1] + len(want):] == 77).all()


def test_png_of_more_slices_than_two_digits_count():
    """Above 64 x 64 slices of 8 KB the checksum's powers take a third digit."""
    import torch
    w, h = 6001, 2000
    rgb = np.random.default_rng(7).integers(0, 256, 3 * w * h).astype(np.uint8)
    want = np.frombuffer(zt.encode_png(rgb, w, h), np.uint8)
    assert len(want) > 64 * 64 * 8192
    d = torch.from_numpy(rgb).cuda()
    out = torch.empty(len(want), dtype=torch.uint8, device="cuda")
    zt.encode_png_device(d.data_ptr(), w, h, out.data_ptr(), len(want))
    assert (out.cpu().numpy() == want).all()
