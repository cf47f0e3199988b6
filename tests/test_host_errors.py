"""The library's host code (csrc/fz_api.cu) on a CUDA runtime that fails where it is told to
(fake_cuda.cu): no GPU, no kernel."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA_ERROR = 719  # cudaErrorLaunchFailure


@pytest.fixture(scope="module")
def api(fz, tmp_path_factory):
    import __graft_entry__ as g
    b = g._load_build_module()
    os.makedirs(b.BUILD, exist_ok=True)
    obj = b.compile_one("fz_api.cu")
    d = tmp_path_factory.mktemp("fake")
    src, so = os.path.join(HERE, "fake_cuda.cpp"), str(d / "libfzhost.so")
    runtime, launchers = str(d / "runtime.o"), str(d / "launchers.o")
    subprocess.check_call(["g++", "-std=c++17", "-fPIC", "-I" + os.path.join(b.cuda_home(), "include"), "-c", src, "-o", runtime])
    subprocess.check_call([b.nvcc()] + b.ARCH + b.NVCC_FLAGS + ["-x", "cu", "-c", src, "-o", launchers])
    subprocess.check_call(["g++", "-shared", "-Wl,-Bsymbolic", "-o", so, obj, runtime, launchers])
    L = C.CDLL(so)
    for name, (res, args) in fz.SIGNATURES.items():
        if hasattr(L, name):
            f = getattr(L, name)
            f.restype, f.argtypes = res, args
    L.fake_calls.restype = C.c_char_p
    L.fake_fail.argtypes = [C.c_char_p, C.c_int, C.c_int]
    return L


@pytest.fixture
def ws(api, fz):
    h = C.c_void_p()
    assert api.fz_workspace_create(1 << 20, C.byref(h)) == fz.SUCCESS
    api.fake_reset()
    yield h
    api.fake_reset()
    api.fz_workspace_destroy(h)


def aligned(n, dtype):
    raw = np.zeros(n * np.dtype(dtype).itemsize + 16, np.uint8)
    off = -raw.ctypes.data % 16
    return raw[off:off + n * np.dtype(dtype).itemsize].view(dtype)


def calls(api):
    return api.fake_calls().decode().split()


@pytest.mark.parametrize("call,nth", [(b"cudaMemcpyAsync", 1), (b"cudaMemcpyAsync", 2), (b"cudaStreamSynchronize", 1)])
def test_scan_encode_total_only_when_read(api, fz, ws, call, nth):
    """The chunk total is stored only after the wait that brought it."""
    n = 4096
    shuffled, flags = aligned(2 * n, np.uint8), aligned(n // 8, np.uint32)
    nnz = C.c_uint64(123456789)
    api.fake_fail(call, nth, CUDA_ERROR)
    st = api.fz_scan_encode(ws, shuffled.ctypes.data, flags.ctypes.data, n, None, None, C.byref(nnz), None)
    assert st != fz.SUCCESS
    assert nnz.value == 123456789
    api.fake_reset()
    assert api.fz_scan_encode(ws, shuffled.ctypes.data, flags.ctypes.data, n, None, None, C.byref(nnz), None) == fz.SUCCESS
    assert nnz.value == 7


@pytest.mark.parametrize("nth", [0, 1, 2, 3])
def test_decompress_host_leaves_no_copy_under_way(api, fz, oracle, ws, nth):
    """Whichever copy fails to start, none of the caller's buffers is in use once the call has returned."""
    x = np.linspace(0, 1, 9000, dtype=np.float32)
    stream = oracle.compress(x, (9000, 1, 1), 1e-3, rel=True, mode=1)
    src, out = aligned(stream.size, np.uint8), np.zeros(x.size, np.float32)
    src[:] = stream
    if nth:
        api.fake_fail(b"cudaMemcpyAsync", nth, CUDA_ERROR)
    st = api.fz_decompress_host(ws, src.ctypes.data, src.size, out.ctypes.data, out.size, None)
    assert (st == fz.SUCCESS) == (nth == 0)
    assert api.fake_pending() == 0


def test_compress_host_leaves_no_copy_under_way(api, fz, ws):
    """A bound that the compression refuses after the field's copy has been enqueued."""
    x, out = aligned(9000, np.float32), aligned(1 << 16, np.uint8)
    st = api.fz_compress_host(ws, x.ctypes.data, x.size, fz.Dims(9000, 1, 1), -1.0, fz.EB_REL, 1, out.ctypes.data, out.size, None, None)
    assert st == fz.INVALID_ARG
    assert api.fake_pending() == 0


def compressed(api, fz, ws, items, rel=True):
    """The launches of one compression of `items` encode items."""
    n = items * 16384
    x, out = aligned(n, np.float32), aligned(fz.max_compressed_bytes(n, (n, 1, 1)), np.uint8)
    api.fake_reset()
    st = api.fz_compress(ws, x.ctypes.data, n, fz.Dims(n, 1, 1), 1e-3, fz.EB_REL if rel else fz.EB_ABS, 1, out.ctypes.data,
                         out.size, None, None)
    assert st == fz.SUCCESS
    return calls(api)


@pytest.mark.parametrize("cluster", [16, 8, 1, 0])
def test_fields_past_the_largest_cluster_of_the_device(api, fz, ws, cluster):
    """A cluster that the device cannot place is not launched: such a field takes the other launches."""
    api.fake_largest_cluster(cluster)
    try:
        for items in (1, 8, 9, 16, 17):
            if items <= cluster:
                assert compressed(api, fz, ws, items) == ["whole"]
            else:
                assert compressed(api, fz, ws, items) == ["range", "encode", "compact"]
                assert compressed(api, fz, ws, items, rel=False) == ["encode", "compact"]
        # in a batch: a field of 20 items takes the range of one of 12 ahead unless that is one cluster
        fields, keep = [], []
        for items in (20, 12):
            n = items * 16384
            x, out = aligned(n, np.float32), aligned(fz.max_compressed_bytes(n, (n, 1, 1)), np.uint8)
            keep += [x, out]
            fields.append({"src": x.ctypes.data, "dst": out.ctypes.data, "n": n, "dims": (n, 1, 1), "eb": 1e-3, "dst_capacity": out.size})
        api.fake_reset()
        assert api.fz_compress_batch(ws, fz.fields_array(fields), 2, fz.EB_REL, 1, None) == fz.SUCCESS
        assert calls(api) == ["range", "encode", "compact"] + (["whole"] if cluster >= 12 else ["encode", "compact"])
    finally:
        api.fake_largest_cluster(16)
