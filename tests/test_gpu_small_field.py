"""Compression without a compaction launch (k_whole_field, csrc/fz_compress.cu) against the oracle,
byte for byte, around its edges: no full block, one block, items of 16384 codes around 1, 2, 8, 15
and 16 of them (the cluster's limit), tails, fields longer than their dims, values past the 16-bit
path; up to and past one resident wave of items, against the list launches too; recorded in a graph;
between larger fields of a batch."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DIMS = [(100, 1, 1), (2047, 1, 1), (2048, 1, 1), (2049, 1, 1), (16384, 1, 1), (16385, 1, 1), (18432, 1, 1),
        (131071, 1, 1), (245761, 1, 1), (262143, 1, 1), (262144, 1, 1), (262145, 1, 1), (32, 64, 1), (128, 128, 1),
        (129, 127, 1), (255, 257, 1), (512, 512, 1), (4096, 64, 1), (4100, 60, 1), (511, 513, 1), (513, 511, 1),
        (16, 16, 8), (25, 26, 27), (64, 64, 64), (63, 65, 64), (64, 65, 64), (400, 3, 200)]


@pytest.fixture(scope="module")
def ws(fz):
    torch.cuda.set_device(0)
    return fz.Workspace(1 << 20)


def field(n, seed, peak=1.0):
    rng = np.random.default_rng(seed)
    return (peak * np.cumsum(rng.standard_normal(n)) / np.sqrt(n)).astype(np.float32)


@pytest.mark.parametrize("dims", DIMS, ids=["x".join(map(str, d)) for d in DIMS])
@pytest.mark.parametrize("extra", [0, 700])
def test_small_streams(fz, oracle, ws, dims, extra):
    n = dims[0] * dims[1] * dims[2] + extra
    for data in (field(n, n), np.abs(field(n, n + 1)), field(n, n + 2, 1e5), np.full(n, 2.5, np.float32)):
        dev = torch.from_numpy(data).cuda()
        rels = data.max() > data.min()
        for eb, rel, mode in ((1e-3, True, 1), (1e-3, True, 0), (1e-5, True, 1), (1e-2, False, 1), (1e-2, False, 0)):
            if rel and not rels:
                continue
            want = oracle.compress(data, dims, eb, rel=rel, mode=mode)
            got = fz.compress(dev, dims, eb, rel=rel, mode=mode, ws=ws)
            assert np.array_equal(got.cpu().numpy(), want), (eb, rel, mode)


def test_small_between_large(fz, oracle, ws):
    """The launch that follows a larger field's, and precedes one, on the same workspace, called,
    in one batch call and recorded in a graph."""
    shapes = [(900, 700, 1), (128, 128, 1), (300000, 1, 1), (64, 64, 64), (100, 1, 1), (70, 80, 90)]
    fields = [field(x * y * z, x) for x, y, z in shapes]
    dev = [torch.from_numpy(f).cuda() for f in fields]
    outs = [torch.zeros(fz.max_compressed_bytes(f.size, d), dtype=torch.uint8, device="cuda") for f, d in zip(fields, shapes)]

    def run():
        for f, d, o in zip(dev, shapes, outs):
            fz.compress(f, d, 1e-3, ws=ws, out=o, readback=False)

    def check():
        torch.cuda.synchronize()
        for f, d, o in zip(fields, shapes, outs):
            want = oracle.compress(f, d, 1e-3, rel=True, mode=1)
            assert np.array_equal(o[:want.size].cpu().numpy(), want), d
            o.zero_()

    run()
    check()
    fz.compress_batch(ws, fz.fields_array([
        {"src": f.data_ptr(), "dst": o.data_ptr(), "n": f.numel(), "dims": d, "eb": 1e-3, "dst_capacity": o.numel()}
        for f, d, o in zip(dev, shapes, outs)]))
    check()
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.stream(stream), torch.cuda.graph(graph, stream=stream):
        run()
    for _ in range(2):
        graph.replay()
        check()


@pytest.mark.parametrize("dims", [(17 * 16384, 1, 1), (152 * 16384 + 5, 1, 1), (608 * 16384, 1, 1), (608 * 16384 + 1, 1, 1),
                                  (2048, 456 * 8, 1), (2047, 456 * 8, 1), (2048, 456 * 8 + 1, 1), (128, 128, 456), (129, 127, 457),
                                  (128, 129, 456)], ids=lambda d: "x".join(map(str, d)))
def test_one_wave(fz, oracle, dims):
    n = dims[0] * dims[1] * dims[2]
    w = fz.Workspace(n)
    for data in (field(n, 1, 50.0), np.abs(field(n, 2)), field(n, 3, 1e5)):
        dev = torch.from_numpy(data).cuda()
        listed = torch.zeros(fz.max_compressed_bytes(n, dims), dtype=torch.uint8, device="cuda")
        for eb, rel, mode in ((1e-3, True, 1), (1e-2, False, 1), (1e-5, True, 0)):
            want = oracle.compress(data, dims, eb, rel=rel, mode=mode)
            got = fz.compress(dev, dims, eb, rel=rel, mode=mode, ws=w)
            assert np.array_equal(got.cpu().numpy(), want), (eb, rel, mode)
            fz.compress_batch(w, fz.fields_array([{"src": dev.data_ptr(), "dst": listed.data_ptr(), "n": n, "dims": dims,
                                                   "eb": eb, "dst_capacity": listed.numel()}]), rel=rel, mode=mode)
            assert np.array_equal(listed[:want.size].cpu().numpy(), want), (eb, rel, mode)
