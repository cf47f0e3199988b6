"""Encode and compaction in one launch after the range launch (k_whole_field<ND, true>): a wait that
gave up marks the stream whichever item it was, launches of several workspaces at the same time, and
the limits of the dispatch, found from the device."""
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ITEM = 16384


def field(n, seed):
    rng = np.random.default_rng(seed)
    return (np.cumsum(rng.standard_normal(n)) / np.sqrt(n)).astype(np.float32)


def wave(nd):
    """Items of one resident wave: 4 CTAs an SM in 1D, 3 otherwise."""
    return torch.cuda.get_device_properties(0).multi_processor_count * (4 if nd == 1 else 3)


def dims_of(nd, items):
    return [(items * ITEM, 1, 1), (256, 64 * items, 1), (64, 64, 4 * items)][nd - 1]


@pytest.mark.parametrize("nd", [1, 2, 3])
@pytest.mark.parametrize("where", ["first", "second", "middle", "last"])
@pytest.mark.parametrize("mode", [0, 1])
def test_given_up_wait_marks_the_stream(fz, oracle, nd, where, mode):
    items = 40
    dims, item = dims_of(nd, items), {"first": 0, "second": 1, "middle": items // 2, "last": items - 1}[where]
    data = field(items * ITEM, nd)
    x, ws = torch.from_numpy(data).cuda(), fz.Workspace(items * ITEM)
    out = torch.zeros(fz.max_compressed_bytes(x.numel(), dims, mode), dtype=torch.uint8, device="cuda")
    want = oracle.compress(data, dims, 1e-3, rel=True, mode=mode)
    for readback in (True, False):
        assert ws.selftest_whole_timeout(x, dims, 1e-3, item, out, mode=mode, readback=readback) == (
            fz.TIMEOUT if readback else fz.SUCCESS)
        torch.cuda.synchronize()
        assert fz.parse_header(out[:64].cpu().numpy()).flags & 2
        with pytest.raises(fz.FzError):
            fz.decompress(out, ws=ws)
        assert ws.status() == (fz.SUCCESS if readback else fz.TIMEOUT)
        # the next call on the workspace is as any other
        got = fz.compress(x, dims, 1e-3, mode=mode, ws=ws, out=out)
        assert np.array_equal(got.cpu().numpy(), want)
        assert fz.parse_header(got[:64].cpu().numpy()).flags & 2 == 0


def test_no_wait_to_give_up(fz):
    """Fields of one cluster, or past one wave, have no such wait; nor does an item past the last."""
    for items, item in ((16, 3), (40, 40), (wave(2) + 1, 3)):
        dims = dims_of(2, items)
        x, ws = torch.ones(items * ITEM, device="cuda"), fz.Workspace(items * ITEM)
        out = torch.zeros(fz.max_compressed_bytes(x.numel(), dims), dtype=torch.uint8, device="cuda")
        assert ws.selftest_whole_timeout(x, dims, 1e-3, item, out) == fz.INVALID_ARG


@pytest.mark.parametrize("nd", [1, 2, 3])
@pytest.mark.parametrize("readback", [True, False])
def test_limits(fz, oracle, nd, readback):
    """One launch up to a wave of items (half a wave where the caller does not wait), the encode and
    compaction launches one item past it; the same bytes."""
    most = wave(nd) if readback else wave(nd) // 2
    data = field((most + 1) * ITEM, nd)
    x, ws = torch.from_numpy(data).cuda(), fz.Workspace(data.size)
    for items in (most, most + 1):
        dims, n = dims_of(nd, items), items * ITEM
        out = torch.zeros(fz.max_compressed_bytes(n, dims), dtype=torch.uint8, device="cuda")
        ws.enable_timing(16)
        fz.compress(x[:n], dims, 1e-3, ws=ws, out=out, readback=readback)
        assert ws.kernel_time("k_compact_fields")[0] == items - most
        ws.enable_timing(0)
        want = oracle.compress(data[:n], dims, 1e-3, rel=True, mode=1)
        assert np.array_equal(out[:want.size].cpu().numpy(), want)


@pytest.mark.parametrize("nd", [1, 2, 3])
def test_several_at_once(fz, oracle, nd):
    """Four threads, each with its own stream and workspace, compress fields of half to one wave (with
    the size read back) and of half a wave (without), all at once: CTAs of several launches wait for
    counts while others of theirs have not started."""
    w = wave(nd)
    jobs = []
    for k, items in enumerate((w // 2 - 1, w * 2 // 3, w * 9 // 10, w)):
        data = field(items * ITEM, 10 * nd + k)
        dims = dims_of(nd, items)
        want = oracle.compress(data, dims, 1e-3, rel=True, mode=1)
        jobs.append((torch.from_numpy(data).cuda(), dims, want, k == 0))
    bad = []
    start = threading.Barrier(len(jobs))

    def work(x, dims, want, deferred):
        try:
            stream, ws = torch.cuda.Stream(), fz.Workspace(x.numel())
            outs = [torch.zeros(fz.max_compressed_bytes(x.numel(), dims), dtype=torch.uint8, device="cuda") for _ in range(8)]
            torch.cuda.synchronize()
            start.wait(60)
            for out in outs:
                fz.compress(x, dims, 1e-3, ws=ws, out=out, stream=stream, readback=not deferred)
            stream.synchronize()
            assert ws.status(stream) == fz.SUCCESS
            for out in outs:
                assert np.array_equal(out[:want.size].cpu().numpy(), want), dims
        except Exception as e:  # into the main thread
            bad.append(e)

    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad


@pytest.mark.parametrize("nd", [1, 2, 3])
def test_largest_cluster(fz, nd):
    """Sixteen items, the range too, in one launch; a range launch from seventeen on."""
    for items in (16, 17):
        dims, n = dims_of(nd, items), items * ITEM
        x, ws = torch.from_numpy(field(n, nd)).cuda(), fz.Workspace(n)
        ws.enable_timing(16)
        fz.compress(x, dims, 1e-3, ws=ws)
        assert ws.kernel_time("k_range_fields")[0] == items - 16
        assert ws.kernel_time("k_encode_fields")[0] == 1
        ws.enable_timing(0)
