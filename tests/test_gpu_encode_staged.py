"""The staged 16-bit encode (csrc/fz_encode.cuh) against the oracle, byte for byte, where it can
go wrong: rows around its limits (8, 64 and 4096 elements, multiples of 4, 2 and 1), items and
tails around 16384 elements, planes shorter than an item, fields longer than their dims, values
on rounding ties of either sign, and magnitudes around the bounds past which it hands an item
or a field to the float path (up to deltas that overflow their codes)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(16384, 1, 1), (16383, 1, 1), (16385, 1, 1), (40961, 1, 1), (100, 1, 1), (67, 1, 1),
          (64, 300, 1), (65, 300, 1), (66, 299, 1), (127, 131, 1), (2049, 17, 1), (4095, 9, 1), (4096, 9, 1),
          (4097, 9, 1), (4100, 9, 1), (4098, 33, 1), (20001, 19, 1), (63, 300, 1),
          (64, 64, 5), (65, 7, 40), (66, 1, 300), (68, 9, 33), (64, 3, 100), (129, 127, 3), (4096, 2, 9), (4099, 3, 9),
          (501, 37, 17), (250, 131, 9), (8, 2100, 1), (9, 2000, 1), (10, 1900, 1), (12, 1500, 1), (17, 1001, 1),
          (33, 500, 1), (62, 290, 1), (8, 8, 60), (9, 5, 400), (13, 1, 1500), (31, 43, 13), (48, 20, 30), (62, 70, 5),
          (7, 900, 1), (6, 50, 70)]


@pytest.fixture(scope="module")
def ws(fz):
    torch.cuda.set_device(0)
    return fz.Workspace(1 << 20)


def check(fz, oracle, ws, data, dims, eb, rel, mode):
    st = fz.compress(torch.from_numpy(data).cuda(), dims, eb, rel=rel, mode=mode, ws=ws)
    want = oracle.compress(data, dims, eb, rel=rel, mode=mode)
    assert np.array_equal(st.cpu().numpy(), want)


@pytest.mark.parametrize("dims", SHAPES, ids=["x".join(map(str, d)) for d in SHAPES])
@pytest.mark.parametrize("extra", [0, 2051])
def test_staged_streams(fz, oracle, ws, dims, extra):
    n = dims[0] * dims[1] * dims[2] + extra
    rng = np.random.default_rng(n)
    half = rng.integers(-200, 201, n)  # multiples of the bound 1/2: every odd one is a rounding tie
    for low, peak in ((-1, 1), (0, 1), (-1, 20), (-1, 75), (0, 330)):
        data = (half * (peak * 0.5)).astype(np.float32)
        if low == 0:
            data = np.abs(data)
        near = np.nextafter(data, np.float32(np.inf) * rng.choice([-1, 1], n).astype(np.float32))
        data = np.where(rng.random(n) < 0.3, near, data).astype(np.float32)
        if low == 0:
            data = np.abs(data)
        for mode in (0, 1):
            check(fz, oracle, ws, data, dims, 0.5, False, mode)
        # a relative bound that is (nearly) 1/2 as well
        check(fz, oracle, ws, data, dims, 0.5 / float(data.max() - data.min()), True, 1)


@pytest.mark.parametrize("dims", [(900, 70, 1), (4101, 11, 1), (70, 30, 21), (501, 37, 17)],
                         ids=["2d", "2d-wide", "3d", "3d-odd"])
@pytest.mark.parametrize("top", [15, 16, 17, 31, 32, 33])
def test_staged_byte_deltas(fz, oracle, ws, dims, top):
    """Deltas around the 8 bits below which a block's planes 8..14 are left out: values of +-top
    give sums of four (2D) and eight (3D) of up to 128 either way, -128 among them."""
    n = dims[0] * dims[1] * dims[2]
    rng = np.random.default_rng(top)
    data = (top * rng.choice([-1, 1], n)).astype(np.float32)
    data[n // 2:] = (data[n // 2:] * rng.integers(0, 2, n - n // 2)).astype(np.float32)
    for mode in (0, 1):
        check(fz, oracle, ws, data, dims, 0.5, False, mode)


@pytest.mark.parametrize("dims", [(40000, 1, 1), (400, 101, 1), (4101, 11, 1), (70, 30, 21)],
                         ids=["1d", "2d", "2d-wide", "3d"])
def test_staged_bounds(fz, oracle, ws, dims):
    """One item past the bound among others, an outlier just below and just above it, and NaN."""
    n = dims[0] * dims[1] * dims[2]
    rng = np.random.default_rng(1)
    base = rng.normal(0, 30, n).astype(np.float32)
    for peak in (4000.0, 4100.0, 8140.0, 8160.0, 16290.0, 16310.0, 32500.0, 32700.0, 66000.0, 3e9):
        data = base.copy()
        data[n // 2] = peak
        check(fz, oracle, ws, data, dims, 0.5, False, 1)
        check(fz, oracle, ws, data, dims, 0.5 / float(data.max() - data.min()), True, 1)
        check(fz, oracle, ws, -data, dims, 0.5 / float(data.max() - data.min()), True, 1)
    data = base.copy()
    data[n // 3] = np.nan
    check(fz, oracle, ws, data, dims, 0.5, False, 1)


@pytest.mark.parametrize("n", [5001, 16387, 40001, (1 << 22) + 3])
def test_nan_before_the_last_elements(fz, ws, n):
    """A NaN in the elements that the threads holding the last n mod 4 elements read before them."""
    w = ws if n <= 1 << 20 else fz.Workspace(n)
    last = (n - 1) // 1024 * 1024
    for pos in {0, 1, last, max(0, last - 1024), max(0, last - 3 * 1024 + 4), last // 16384 * 16384}:
        x = np.linspace(0, 1, n, dtype=np.float32)
        x[pos] = np.nan
        with pytest.raises(fz.FzError) as e:
            fz.compress(torch.from_numpy(x).cuda(), (n, 1, 1), 1e-3, rel=True, ws=w)
        assert e.value.status == fz.NONFINITE_INPUT, pos
