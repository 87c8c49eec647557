"""Flat morphology on the GPU: bit-identical (NaN and signed zeros included) to the reference's
erode / dilate, through its golden vectors and the oracle."""
from __future__ import annotations

import zlib

import numpy as np
import pytest

import iane_gb300
import oracle
from golden_cases import morph_cases
from gpu_helpers import empty_like_np, to_gpu, to_host, torch

pytestmark = pytest.mark.gpu


def run_gpu(src, radius, op, border, mask=None):
    out = empty_like_np(src.shape, src.dtype)
    fp = None if mask is None else to_gpu(mask.astype(np.uint8))
    iane_gb300.morphology(to_gpu(src), out, radius, op, border, fp)
    return to_host(out)


def test_known_answers(cuda):
    # test/unit/algorithms/color_morphology_cases.hpp:87-117 (a crop of a 6-element image)
    t = torch()
    src = to_gpu(np.array([99, 3, 1, 5, 2, 99], np.int32))[1:5]
    out = t.zeros(4, dtype=t.int32, device="cuda")
    forward = to_gpu(np.array([0, 0, 1], np.uint8))
    for op, fp, border, want in (("erode", None, "clamp", [1, 1, 1, 2]), ("dilate", None, "clamp", [3, 5, 5, 5]),
                                 ("erode", forward, "zero", [1, 5, 2, 0]), ("dilate", forward, "zero", [0, 3, 1, 5])):
        iane_gb300.morphology(src, out, (1,), op, border, fp)
        assert to_host(out).tolist() == want, (op, border)


@pytest.mark.parametrize("case", morph_cases(), ids=lambda c: c[0])
def test_golden(cuda, case):
    name, src, radius, op, border, mask, expected = case
    assert run_gpu(src, radius, op, border, mask).tobytes() == expected.tobytes(), name


TYPES = [np.uint8, np.int8, np.uint16, np.int16, np.int32, np.uint32, np.float32, np.float64]


@pytest.mark.parametrize("dtype", TYPES, ids=lambda d: np.dtype(d).name)
@pytest.mark.parametrize("shape,radius", [((200,), (5,)), ((37, 70), (2, 3)), ((9, 40, 45), (1, 2, 3)),
                                          ((3, 5, 4), (2, 0, 4)), ((64, 300), (40, 1))])
def test_box_parity(cuda, dtype, shape, radius):
    rng = np.random.default_rng(zlib.crc32(repr((np.dtype(dtype).name, shape)).encode()))
    if np.issubdtype(dtype, np.floating):
        src = rng.standard_normal(shape).astype(dtype)
        src[rng.random(shape) < 0.05] = np.nan
        src[rng.random(shape) < 0.05] = 0.0
        src[rng.random(shape) < 0.05] = -0.0
    else:
        info = np.iinfo(dtype)
        src = rng.integers(info.min, info.max, shape, dtype=dtype, endpoint=True)
    for op in ("erode", "dilate"):
        for border in ("clamp", "zero", "mirror"):
            ref = np.zeros_like(src)
            oracle.morphology(src, ref, radius, op, border)
            assert run_gpu(src, radius, op, border).tobytes() == ref.tobytes(), (op, border)


@pytest.mark.parametrize("shape,radius", [((30, 41), (2, 3)), ((7, 12, 15), (1, 2, 1))])
def test_masked_footprints(cuda, shape, radius):
    rng = np.random.default_rng(len(shape))
    src = rng.integers(0, 1000, shape).astype(np.int32)
    mask = rng.random(tuple(2 * r + 1 for r in radius)) < 0.4
    for op in ("erode", "dilate"):
        for border in ("clamp", "zero", "mirror"):
            ref = np.zeros_like(src)
            oracle.morphology(src, ref, radius, op, border, mask)
            assert np.array_equal(run_gpu(src, radius, op, border, mask), ref), (op, border)


@pytest.mark.parametrize("op", ["opening", "closing"])
def test_compound_in_place_and_strided(cuda, op):
    t = torch()
    rng = np.random.default_rng(3)
    big = rng.integers(0, 256, (10, 40, 60), dtype=np.uint8)
    src_np = np.ascontiguousarray(big[1:9, 3:37, 5:55])
    ref = np.zeros_like(src_np)
    oracle.morphology(src_np, ref, (1, 2, 2), op, "clamp")
    g = to_gpu(big)
    view = g[1:9, 3:37, 5:55]
    iane_gb300.morphology(view, view, (1, 2, 2), op, "clamp")  # in place on a strided crop
    assert np.array_equal(to_host(view), ref)
    assert np.array_equal(to_host(g)[0], big[0])  # outside the crop untouched
    # the reference's 4-D slab-and-impulse case, in 3-D
    img = np.zeros((3, 3, 4), np.int32)
    img[:, :, :2] = 1
    img[1, 1, 3] = 1
    close = op == "closing"
    if close:
        img = 1 - img
    out = empty_like_np(img.shape, np.int32)
    iane_gb300.morphology(to_gpu(img), out, (1, 1, 1), op)
    want = np.zeros_like(img)
    want[:, :, :2] = 1
    assert np.array_equal(to_host(out), 1 - want if close else want)
    del t


def test_errors(cuda):
    a = to_gpu(np.zeros((8, 8), np.float32))
    with pytest.raises(iane_gb300.IaneInvalidArgument):
        iane_gb300.morphology(a, a.clone(), (-1, 1))
    with pytest.raises(iane_gb300.IaneInvalidArgument):
        iane_gb300.morphology(a, to_gpu(np.zeros((8, 8), np.float64)), (1, 1))
    with pytest.raises(iane_gb300.IaneError) as info:
        iane_gb300.morphology(a, a.clone(), (600, 600), footprint=None)  # direct-kernel work bound
    assert info.value.status == iane_gb300.abi.UNSUPPORTED
    with pytest.raises(iane_gb300.IaneError):
        iane_gb300.morphology(to_gpu(np.zeros((8, 8), np.float32)).bfloat16(), a.clone().bfloat16(), (1, 1))


@pytest.mark.parametrize("radius", [1, 2, 3])
@pytest.mark.parametrize("dtype", [np.uint8, np.int16, np.uint32, np.float32, np.float64], ids=lambda d: np.dtype(d).name)
def test_cube_footprints(cuda, dtype, radius):
    """Equal radii on all three axes take the unrolled kernel with the z window in registers;
    several z chunks (the volume is deeper than one chunk), NaN and signed zeros included."""
    rng = np.random.default_rng(zlib.crc32(repr((np.dtype(dtype).name, radius)).encode()))
    shape = (45, 37, 70)
    if np.issubdtype(dtype, np.floating):
        src = rng.standard_normal(shape).astype(dtype)
        src[rng.random(shape) < 0.05] = np.nan
        src[rng.random(shape) < 0.05] = 0.0
        src[rng.random(shape) < 0.05] = -0.0
    else:
        info = np.iinfo(dtype)
        src = rng.integers(info.min, info.max, shape, dtype=dtype, endpoint=True)
    r = (radius,) * 3
    for op in ("erode", "dilate"):
        for border in ("clamp", "zero", "mirror"):
            ref = np.zeros_like(src)
            oracle.morphology(src, ref, r, op, border)
            assert run_gpu(src, r, op, border).tobytes() == ref.tobytes(), (op, border)


@pytest.mark.parametrize("radius", [1, 2, 3])
def test_cube_footprints_on_strided_views(cuda, radius):
    """The cube kernel's per-block staging offsets on a cropped view with an x stride of two
    elements, all three borders."""
    t = torch()
    rng = np.random.default_rng(100 + radius)
    big = rng.standard_normal((44, 33, 140)).astype(np.float32)
    big[rng.random(big.shape) < 0.03] = np.nan
    crop = (slice(2, 40), slice(3, 30), slice(1, 130, 2))
    src = np.ascontiguousarray(big[crop])
    g = to_gpu(big)
    r = (radius,) * 3
    for op in ("erode", "dilate"):
        for border in ("clamp", "zero", "mirror"):
            ref = np.zeros_like(src)
            oracle.morphology(src, ref, r, op, border)
            out = t.zeros((44, 33, 140), dtype=t.float32, device="cuda")
            iane_gb300.morphology(g[crop], out[crop], r, op, border)
            assert to_host(out[crop]).tobytes() == ref.tobytes(), (op, border)


def test_cube_footprint_with_a_plane_beyond_31_bit_offsets(cuda):
    """A view whose plane spans more than 2^31 bytes (two rows 2^31 + 4 KiB apart) takes the
    general fused 3-D kernel; the result is the same."""
    t = torch()
    row = (1 << 29) + 1024  # elements between the two rows: 2^31 + 4 KiB
    buf = t.zeros(row + 3 * 64 + 64, dtype=t.float32, device="cuda")
    rng = np.random.default_rng(7)
    vals = rng.standard_normal((3, 2, 64)).astype(np.float32)
    view = buf.as_strided((3, 2, 64), (64, row, 1))
    view.copy_(t.from_numpy(vals).cuda())
    out = t.zeros((3, 2, 64), dtype=t.float32, device="cuda")
    for op in ("erode", "dilate"):
        ref = np.zeros_like(vals)
        oracle.morphology(vals, ref, (1, 1, 1), op, "clamp")
        iane_gb300.morphology(view, out, (1, 1, 1), op, "clamp")
        assert to_host(out).tobytes() == ref.tobytes(), op
    del buf


@pytest.mark.parametrize("dtype", [np.uint8, np.int8, np.uint16, np.int16, np.float32], ids=lambda d: np.dtype(d).name)
@pytest.mark.parametrize("shape,radius", [
    ((1, 1), (1, 1)), ((9, 7), (4, 4)),            # everything is border
    ((8, 24), (1, 2)), ((17, 31), (2, 1)),         # one thread inside a row; an odd tail
    ((33, 263), (3, 3)), ((40, 256), (0, 4)),      # several warps, a row's last element alone; whole groups
    ((5, 19, 530), (0, 2, 1)),                     # a stack of planes
    ((700, 2101), (4, 3)), ((640, 1024), (3, 4)),  # radii of 3 and 4 on larger images (integers; f32)
])
def test_planes_of_packed_rows(cuda, dtype, shape, radius):
    # rows of every alignment: the packed image, and a crop whose rows start one element in
    rng = np.random.default_rng(zlib.crc32(repr((np.dtype(dtype).name, shape, radius)).encode()))
    wide = (*shape[:-1], shape[-1] + 2)
    if dtype == np.float32:
        big = rng.standard_normal(wide).astype(dtype)
        for value in (np.nan, 0.0, -0.0, np.inf):
            big[rng.random(wide) < 0.05] = value
    else:
        info = np.iinfo(dtype)
        big = rng.integers(info.min, info.max, wide, dtype=dtype, endpoint=True)
    for op in ("erode", "dilate"):
        for border in ("clamp", "zero", "mirror"):
            src = np.ascontiguousarray(big[..., 1:-1])
            ref = np.zeros_like(src)
            oracle.morphology(src, ref, radius, op, border)
            assert run_gpu(src, radius, op, border).tobytes() == ref.tobytes(), (op, border)
            g, out = to_gpu(big), to_gpu(np.zeros_like(big))
            iane_gb300.morphology(g[..., 1:-1], out[..., 1:-1], radius, op, border)
            got = to_host(out)
            assert np.ascontiguousarray(got[..., 1:-1]).tobytes() == ref.tobytes(), (op, border, "crop")
            assert not got[..., 0].any() and not got[..., -1].any()


@pytest.mark.parametrize("shape,radius", [
    ((5, 16, 16), 2), ((1, 17, 20), 1),       # one warp; one plane, a row beyond whole groups of rows
    ((9, 33, 260), 2), ((40, 20, 128), 1),    # a third warp of one group; several chunks of planes
    ((17, 120, 132), 3), ((33, 64, 130), 3),  # the widest window; rows that TMA cannot address
])
def test_volumes_of_aligned_rows(cuda, shape, radius):
    # NaN, infinities and zeros of both signs: a warp takes the exact form in planes that hold a -0
    rng = np.random.default_rng(sum(shape) + radius)
    src = rng.standard_normal(shape).astype(np.float32)
    for value in (np.nan, np.inf, -np.inf, 0.0):
        src[rng.random(shape) < 0.03] = value
    half = src.copy()
    src[rng.random(shape) < 0.03] = -0.0
    half[:1 + shape[0] // 2][rng.random((1 + shape[0] // 2, *shape[1:])) < 0.1] = -0.0  # planes with and without
    half = np.where(np.abs(half) < 1.0, np.copysign(np.float32(0), half), half)
    wide = np.zeros((*shape[:-1], shape[-1] + 8), np.float32)
    for data in (src, half):
        wide[..., 4:-4] = data
        for op in ("erode", "dilate"):
            for border in ("clamp", "zero", "mirror"):
                ref = np.zeros_like(data)
                oracle.morphology(data, ref, (radius,) * 3, op, border)
                assert run_gpu(data, (radius,) * 3, op, border).tobytes() == ref.tobytes(), (op, border)
                out = to_gpu(np.zeros((*shape[:-1], shape[-1] + 1), np.float32))
                iane_gb300.morphology(to_gpu(wide)[..., 4:-4], out[..., 1:], (radius,) * 3, op, border)
                got = to_host(out)
                assert np.ascontiguousarray(got[..., 1:]).tobytes() == ref.tobytes(), (op, border, "crop")
                assert not got[..., 0].any()


@pytest.mark.parametrize("dtype", [np.uint8, np.int16, np.float32], ids=lambda d: np.dtype(d).name)
@pytest.mark.parametrize("shape,radius", [
    ((600, 3), (2, 1)), ((2500, 12), (3, 3)),     # blocks of one and of two to four threads side by side
    ((1500, 60), (1, 3)), ((1500, 100), (4, 4)),  # of eight; as narrow as a rule's limit
    ((2000, 300), (1, 2)), ((900, 516), (4, 4)),  # of eight and sixteen beyond whole blocks
    ((70, 4100), (2, 2)),                         # an image lower than the tallest blocks
])
def test_planes_of_narrow_images(cuda, dtype, shape, radius):
    rng = np.random.default_rng(zlib.crc32(repr((np.dtype(dtype).name, shape, radius)).encode()))
    if dtype == np.float32:
        src = rng.standard_normal(shape).astype(dtype)
        for value in (np.nan, 0.0, -0.0, -np.inf):
            src[rng.random(shape) < 0.05] = value
    else:
        info = np.iinfo(dtype)
        src = rng.integers(info.min, info.max, shape, dtype=dtype, endpoint=True)
    for op, border in (("erode", "clamp"), ("dilate", "zero"), ("erode", "mirror")):
        ref = np.zeros_like(src)
        oracle.morphology(src, ref, radius, op, border)
        assert run_gpu(src, radius, op, border).tobytes() == ref.tobytes(), (op, border)


@pytest.mark.parametrize("shape,radius", [
    ((9, 33, 100), 2), ((12, 20, 97), 1), ((8, 41, 250), 3),   # 32 lanes side by side
    ((40, 17, 64), 1), ((7, 21, 65), 2), ((33, 64, 184), 3),   # 16
])
def test_volumes_by_lanes(cuda, shape, radius):
    # rows that end inside a lane's columns and at them, at TMA's pitch
    rng = np.random.default_rng(sum(shape) + radius)
    wide = rng.standard_normal((*shape[:-1], shape[-1] + 8 + -shape[-1] % 4)).astype(np.float32)
    for value in (np.nan, np.inf, 0.0):
        wide[rng.random(wide.shape) < 0.03] = value
    wide[: shape[0] // 2][rng.random((shape[0] // 2, *wide.shape[1:])) < 0.03] = -0.0
    src = np.ascontiguousarray(wide[..., 4:4 + shape[-1]])
    for op in ("erode", "dilate"):
        for border in ("clamp", "zero", "mirror"):
            ref = np.zeros_like(src)
            oracle.morphology(src, ref, (radius,) * 3, op, border)
            out = empty_like_np(shape, np.float32)
            iane_gb300.morphology(to_gpu(wide)[..., 4:4 + shape[-1]], out, (radius,) * 3, op, border)
            assert to_host(out).tobytes() == ref.tobytes(), (op, border)
