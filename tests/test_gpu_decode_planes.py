"""The fused decompression kernels against the oracle, bit for bit, where their decode changes
method: deltas around the 2^7 below which planes 7..14 are not fetched (per warp), in 1D around
the 2^9 below which sums are packed, deltas up to the code limit, rows whose codes start anywhere in a 4-code group, windows and whole-row spans
around their limits, bands and slabs cut short by the field's end, and tails in the sidecar."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(4096, 1, 1), (12345, 1, 1), (3000, 17, 1), (961, 33, 1), (1921, 16, 1), (130, 50, 1), (67, 131, 1), (5, 700, 1),
          (64, 64, 9), (65, 31, 17), (66, 9, 8), (127, 24, 3), (500, 16, 9), (501, 17, 8), (516, 9, 10), (960, 8, 8),
          (961, 9, 3), (1003, 16, 2), (13, 100, 40), (8, 8, 200)]


@pytest.fixture(scope="module")
def ws(fz):
    torch.cuda.set_device(0)
    return fz.Workspace(1 << 20)


@pytest.mark.parametrize("dims", SHAPES, ids=["x".join(map(str, d)) for d in SHAPES])
@pytest.mark.parametrize("extra", [0, 900])
def test_decode_magnitudes(fz, oracle, ws, dims, extra):
    n = dims[0] * dims[1] * dims[2] + extra
    rng = np.random.default_rng(n)
    for top, share in ((3, 1.0), (31, 1.0), (63, 1.0), (65, 1.0), (127, 1.0), (128, 1.0), (255, 1.0), (257, 1.0), (5000, 0.001), (16000, 0.02), (32767, 0.3)):
        # values whose deltas are mostly small and reach `top` (and beyond it, in sums of neighbours)
        data = np.where(rng.random(n) < share, rng.integers(-top, top + 1, n), rng.integers(-1, 2, n)).astype(np.float32)
        for mode in (0, 1):
            want = oracle.compress(data, dims, 0.5, rel=False, mode=mode)
            st = torch.from_numpy(want.copy()).cuda()
            h = fz.parse_header(want[: fz.HEADER_BYTES])
            got = fz.decompress(st, header=h, ws=ws).cpu().numpy()
            assert np.array_equal(got.view(np.uint32), oracle.decompress(want).view(np.uint32)), (top, mode)
