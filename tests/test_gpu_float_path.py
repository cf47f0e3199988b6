"""The encode's float path (block1d, block2d_ahead, csrc/fz_compress.cuh) against the oracle, byte for
byte: rows below, at and above the 128 elements of a group row, rows that end inside one, bounds too
fine for the 16-bit path, codes that overflow."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DIMS = [(2048, 1, 1), (40000, 1, 1), (300001, 1, 1), (4, 9000, 1), (12, 3000, 1), (64, 700, 1), (124, 500, 1), (128, 500, 1),
        (132, 500, 1), (252, 333, 1), (2044, 41, 1), (4096, 33, 1), (8200, 20, 1), (256, 2000, 1)]


@pytest.mark.parametrize("dims", DIMS, ids=["x".join(map(str, d)) for d in DIMS])
def test_float_path_streams(fz, oracle, dims):
    n = dims[0] * dims[1]
    w = fz.Workspace(n)
    rng = np.random.default_rng(n)
    smooth = np.cumsum(rng.standard_normal(n)).astype(np.float32)
    for data, eb in ((smooth, 1e-5), (smooth, 1e-6), (rng.uniform(-1, 1, n).astype(np.float32), 1.6e-5)):
        x = torch.from_numpy(data).cuda()
        for mode in (0, 1):
            want = oracle.compress(data, dims, eb, rel=True, mode=mode)
            assert np.array_equal(fz.compress(x, dims, eb, mode=mode, ws=w).cpu().numpy(), want), (eb, mode)
            eb_abs = eb * float(data.max() - data.min())
            want = oracle.compress(data, dims, eb_abs, rel=False, mode=mode)
            assert np.array_equal(fz.compress(x, dims, eb_abs, rel=False, mode=mode, ws=w).cpu().numpy(), want), (eb, mode)
