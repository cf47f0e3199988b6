"""The workloads whose speed this repository looks after: compression and decompression of
float32 fields through the package's public entry points.

Fields stand in for the scientific data the path is made for (climate, detector images,
cloud fraction, 1D series): the shapes are those of the benchmark and of the mixed batch
(64 KB to 256 MB a field, 1D/2D/3D, relative bounds 1e-2 to 1e-4), the values are seeded
synthetic ones.  Streams are bytes and have no value in 64 bits; a reconstruction's is the
quantised field times the bin width.
"""
import importlib.util
import math
import os
import sys

import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "fz-gpu_gb300")


def _package():
    if "fz_gpu_gb300" not in sys.modules:
        spec = importlib.util.spec_from_file_location("fz_gpu_gb300", os.path.join(_PKG, "__init__.py"),
                                                      submodule_search_locations=[_PKG])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["fz_gpu_gb300"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["fz_gpu_gb300"]


# op:   compress (stream-ordered, no size readback), compress-size (with it, the default),
#       decompress, roundtrip, call (the default arguments both ways: sizes and headers read
#       back), stages (the reference's own stages one by one), host (host buffers both ways),
#       batch (a graph of many fields, both ways)
# kind: smooth (sums of waves with a patch of zeros, from 0 up), peaks (noise around zero
#       with narrow high peaks), offset (smooth, far from zero: temperatures, pressures)
def _case(op, kind, x, y=1, z=1, eb=1e-3, rel=True, sidecar=True, extra=0, name=None):
    c = {"op": op, "kind": kind, "x": x, "y": y, "z": z, "eb": eb, "rel": rel, "sidecar": sidecar, "extra": extra}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest field of the mixed batch, the plainest call: launches, readbacks and
        # host work are all there is
        _case("call", "smooth", 128, 128, name="call_2d_128x128"),
        # one climate field, compressed by the default call, which returns the size
        _case("compress-size", "smooth", 3600, 1800, name="compress_2d_3600x1800"),
        # a detector image, compressed in stream order (the caller reads sizes later)
        _case("compress", "peaks", 39200, 388, name="compress_2d_39200x388"),
        # the same image at the finer bound, decompressed
        _case("decompress", "peaks", 39200, 388, eb=1e-4, name="decompress_2d_39200x388"),
        # a 3D cloud field, each direction
        _case("compress", "smooth", 500, 500, 100, name="compress_3d_500x500x100"),
        _case("decompress", "smooth", 500, 500, 100, name="decompress_3d_500x500x100"),
        # rows that are not a multiple of anything, both directions, fine bound, off zero
        _case("roundtrip", "offset", 501, 500, 100, eb=1e-4, name="roundtrip_3d_501x500x100"),
        # the same in 2D, in the reference's exact stream (no sidecar) under an absolute bound,
        # with a file longer than its dims
        _case("compress", "smooth", 3601, 1801, eb=5e-4, rel=False, sidecar=False, extra=77,
              name="compat_2d_3601x1801"),
        # a long 1D series, both directions
        _case("roundtrip", "smooth", 1 << 25, name="roundtrip_1d_2p25"),
        # a caller of the reference's separate stages
        _case("stages", "smooth", 3600, 1800, name="stages_2d_3600x1800"),
        # the command line's path: pinned host buffers, both directions
        _case("host", "smooth", 3600, 1800, name="host_2d_3600x1800"),
        # a batch of mixed fields, 64 KB to 256 MB, replayed from one graph
        {"name": "batch_mixed_24", "op": "batch", "count": 24, "mix": 3},
    ]


def draw(rng):
    most = max(work(c)["bytes"] for c in listed())
    while True:
        c = _any(rng)
        if work(c)["bytes"] <= most:
            return c


def _any(rng):
    op = rng.choice(["call", "compress-size", "compress", "compress", "decompress", "decompress", "roundtrip",
                     "stages", "host", "batch"])
    if op == "batch":
        return {"op": op, "count": rng.randint(6, 20), "mix": rng.randint(10, 10 ** 6)}
    n = int(math.exp(rng.uniform(math.log(1 << 14), math.log((1 << 23) if op == "host" else (1 << 26)))))
    nd = rng.choice([1, 2, 2, 3, 3])
    x, y, z = _dims(n, nd, rng.random(), rng.choice([1, 1, 4, 16]))
    kind = rng.choice(["smooth", "offset"] + (["peaks"] if nd == 2 else []))
    sidecar = op not in ("compress", "compress-size") or rng.random() < 0.75
    return _case(op, kind, x, y, z, eb=rng.choice([1e-2, 1e-3, 1e-4]), rel=op == "stages" or rng.random() < 0.8,
                 sidecar=sidecar, extra=rng.choice([0, 0, rng.randint(1, 3000)]) if op != "stages" else 0)


def _dims(n, nd, u, step):
    """x, y, z with about n elements; x a multiple of `step`; u in [0, 1) picks the aspect."""
    if nd == 1:
        return max(64, n), 1, 1
    if nd == 2:
        x = math.sqrt(n) * math.exp((u - 0.3) * 4)
    else:
        x = n ** (1 / 3) * math.exp((u - 0.5) * 2)
    x = max(8, int(x) // step * step)
    if nd == 2:
        return x, max(2, n // x), 1
    y = max(2, int(math.sqrt(n / x)))
    return x, y, max(2, n // (x * y))


def _members(case):
    """The fields of a batch: sizes log-uniform from 64 KB to 256 MB, as cases of one field."""
    import random
    rng = random.Random(case["mix"])
    out = []
    for _ in range(case["count"]):
        n = int(math.exp(rng.uniform(math.log(1 << 14), math.log(1 << 26))))
        nd = rng.choice([1, 2, 3])
        x, y, z = _dims(n, nd, rng.random(), rng.choice([1, 4]))
        kind = rng.choice(["smooth", "peaks"]) if nd == 2 else "smooth"
        out.append(_case("roundtrip", kind, x, y, z, eb=rng.choice([1e-2, 1e-3, 1e-4])))
    return out


def _n(case):
    return case["x"] * case["y"] * case["z"] + case["extra"]


# Stream bytes per element by bound (measured once on these fields; a path cannot know them before
# it has run), smooth and offset fields by number of dimensions.
_STREAM = {1: {1e-2: 0.64, 1e-3: 1.05, 5e-4: 1.18, 1e-4: 1.44}, 2: {1e-2: 0.34, 1e-3: 0.66, 5e-4: 0.78, 1e-4: 1.06},
           3: {1e-2: 0.38, 1e-3: 0.47, 5e-4: 0.54, 1e-4: 0.77},
           "peaks": {1e-2: 0.05, 1e-3: 0.09, 5e-4: 0.1, 1e-4: 0.39}}


def work(case):
    """Each direction reads its input once and writes its output once: 4 bytes an element on the
    field's side, the stream on the other.  Operations: a multiplication and a rounding an
    element, and the differences (sums) along each dimension."""
    if case["op"] == "batch":
        parts = [work(m) for m in _members(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n = _n(case)
    nd = 1 if case["y"] == case["z"] == 1 else 2 if case["z"] == 1 else 3
    stream = _STREAM["peaks" if case["kind"] == "peaks" else nd][case["eb"]] * n
    if case["op"] == "stages":
        # floats to codes; codes to shuffled codes and 5 bytes of flags per 16; shuffled codes and
        # flags to prefix sums and chunks; codes to floats
        return {"bytes": (4 + 2) * n + (2 + 2 + 0.5 + 1 / 64) * n + (2 + 0.5 + 0.5) * n + stream + (2 + 4) * n,
                "flops": 2 * (2 + nd) * n}
    ways = 1 if case["op"] in ("compress", "compress-size", "decompress") else 2
    return {"bytes": ways * (4 * n + stream), "flops": ways * (2 + nd) * n}


# ------------------------------------------------------------------ inputs
def _field(case, seed):
    """The case's field on the GPU, flat, from the seed alone; `extra` elements past its dims."""
    x, y, z = case["x"], case["y"], case["z"]
    dev = torch.device("cuda")
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    h = torch.Generator()
    h.manual_seed(seed)

    def u(lo, hi):
        return lo + (hi - lo) * float(torch.rand(1, generator=h))

    n = x * y * z
    if case["kind"] == "peaks":
        f = 0.5 * torch.randn(1, 1, y, x, generator=g, device=dev)
        # one peak in each of `count` stretches of the image, so that no two fall together
        count = max(1, n * 2000 // (39200 * 388))
        stretch = n // count
        at = torch.arange(count, device=dev) * stretch
        at = at + (torch.rand(count, generator=g, device=dev) * stretch).long().clamp(max=stretch - 1)
        p = torch.zeros(n, device=dev)
        p[at] = torch.exp(math.log(10.0) + math.log(1e3) * torch.rand(count, generator=g, device=dev))
        p = p.view(1, 1, y, x)
        for _ in range(2):
            p = torch.nn.functional.avg_pool2d(p, 3, 1, 1) * 3
        f = (f + p).view(-1)
    else:
        ax = [torch.arange(m, device=dev, dtype=torch.float32) for m in (x, y, z)]
        f = torch.zeros(z, y, x, device=dev)
        for _ in range(6):
            lo, hi = (30.0, 5000.0) if y == z == 1 else (40.0, 800.0)
            waves = [torch.sin(a * (2 * math.pi / math.exp(u(math.log(lo), math.log(hi)))) + u(0, 6.28)) for a in ax]
            if z > 1:
                f += u(0.2, 1.0) * waves[2][:, None, None] * (waves[1][:, None] * waves[0][None, :])[None]
            elif y > 1:
                f += u(0.2, 1.0) * (waves[1][:, None] * waves[0][None, :])[None]
            else:
                f += u(0.2, 1.0) * waves[0][None, None]
        f = f.view(-1)
        lo = float(f.min())
        f = (f - lo) / max(float(f.max()) - lo, 1e-30)
        if case["z"] == 1:
            f += 1e-4 * torch.randn(n, generator=g, device=dev)
        f = torch.clamp(f - 0.35, min=0.0)
        if case["kind"] == "offset":
            f = f + 2.0
    if case["extra"]:
        f = torch.cat([f, torch.linspace(0, 1, case["extra"], device=dev) + f[-1]])
    return f.contiguous()


def _dims_of(case):
    return case["x"], case["y"], case["z"]


def _bound(case, f):
    """The bound of the call: relative as it is, absolute as that share of a field from 0 to 1
    (of noise with peaks: of its own range)."""
    if case["rel"] or case["kind"] != "peaks":
        return case["eb"]
    return case["eb"] * float(f.max() - f.min())


def _abs_bound(case, f):
    """The absolute bound that a relative one stands for: range in 32 bits, times it in 64."""
    return _bound(case, f) if not case["rel"] else case["eb"] * float(f.max() - f.min())


def prepare(case, seed):
    fz = _package()
    if case["op"] == "batch":
        return _prepare_batch(fz, case, seed)
    f = _field(case, seed)
    n, dims = _n(case), _dims_of(case)
    mode = fz.MODE_SIDECAR if case["sidecar"] else fz.MODE_COMPAT
    s = {"fz": fz, "op": case["op"], "x": f, "n": n, "dims": dims, "eb": _bound(case, f), "rel": case["rel"],
         "mode": mode, "ws": fz.Workspace(n)}
    if case["op"] == "stages":
        s["eb"] = _abs_bound(case, f)
        s["chunks"] = torch.zeros(512 * ((n + 255) // 256), dtype=torch.uint8, device=f.device)
        return s
    if case["op"] == "host":
        # pinned buffers, as a program that streams fields through the GPU keeps them
        cap = fz.max_compressed_bytes(n, dims, mode)
        s["x"] = f.cpu().pin_memory().numpy()
        s["out"] = torch.zeros(cap, dtype=torch.uint8).pin_memory().numpy()
        s["rec"] = torch.zeros(n, dtype=torch.float32).pin_memory().numpy()
        return s
    s["out"] = torch.zeros(fz.max_compressed_bytes(n, dims, mode), dtype=torch.uint8, device=f.device)
    if case["op"] in ("decompress", "roundtrip"):
        stream = fz.compress(f, dims, s["eb"], rel=s["rel"], mode=mode, ws=s["ws"])
        s["header"] = fz.parse_header(stream[: fz.HEADER_BYTES].cpu().numpy())
        s["rec"] = torch.zeros(n, dtype=torch.float32, device=f.device)
        if case["op"] == "decompress":
            s["stream"] = stream.clone()
            del s["x"], s["out"]
    return s


def _prepare_batch(fz, case, seed):
    members = _members(case)
    s = {"fz": fz, "op": "batch", "x": [], "out": [], "rec": []}
    comp, dec, most = [], [], max(_n(m) for m in members)
    s["ws"] = ws = fz.Workspace(most)
    for i, m in enumerate(members):
        f = _field(m, seed * 1000 + i)
        n, dims = _n(m), _dims_of(m)
        out = torch.zeros(fz.max_compressed_bytes(n, dims), dtype=torch.uint8, device=f.device)
        rec = torch.zeros(n, dtype=torch.float32, device=f.device)
        stream = fz.compress(f, dims, m["eb"], ws=ws, out=out)
        head = fz.parse_header(stream[: fz.HEADER_BYTES].cpu().numpy())
        s["x"].append(f), s["out"].append(out), s["rec"].append(rec)
        comp.append({"src": f.data_ptr(), "dst": out.data_ptr(), "n": n, "dims": dims, "eb": m["eb"],
                     "dst_capacity": out.numel()})
        dec.append({"src": out.data_ptr(), "dst": rec.data_ptr(), "n": n, "dims": dims, "dst_capacity": n,
                    "src_bytes": out.numel(), "header": head})
    # the schedule the autotuner picks for mixed batches: list launches, 16 branches
    s["batch"] = fz.Batch.scheduled(ws, fz.fields_array(comp), fz.fields_array(dec), fz.Schedule(16, 1))
    return s


def run(s):
    """One pass.  A stream is returned in its buffer, whose bytes past the stream stay zero; its size
    beside it where the call reads it back."""
    fz, op = s["fz"], s["op"]
    if op == "batch":
        s["batch"].launch()
        return {"streams": s["out"], "fields": s["rec"]}
    if op == "stages":
        codes = fz.lorenzo_construct(s["x"], s["dims"], s["eb"])
        shuffled, bits, flags = fz.bitshuffle_flag(codes)
        sums, chunks, nnz = fz.scan_encode(shuffled, flags, s["n"], ws=s["ws"])
        s["chunks"][: chunks.numel()].copy_(chunks)  # into the buffer that the caller keeps
        field = fz.lorenzo_reconstruct(codes, s["dims"], s["eb"])
        return {"codes": codes, "shuffled": shuffled, "bits": bits, "flags": flags, "sums": sums,
                "chunks": s["chunks"], "nnz": nnz, "field": field}
    if op == "host":
        stream = fz.compress_host(s["x"], s["dims"], s["eb"], rel=s["rel"], mode=s["mode"], ws=s["ws"],
                                  out_np=s["out"])
        field = fz.decompress_host(stream, ws=s["ws"], out_np=s["rec"])
        return {"stream": s["out"], "size": stream.size, "field": field}
    if op == "decompress":
        return {"field": fz.decompress(s["stream"], header=s["header"], out=s["rec"], ws=s["ws"])}
    size = op in ("call", "compress-size")
    stream = fz.compress(s["x"], s["dims"], s["eb"], rel=s["rel"], mode=s["mode"], ws=s["ws"], out=s["out"],
                         readback=size)
    out = {"stream": s["out"]}
    if size:
        out["size"] = stream.numel()
    if op == "call":
        out["field"] = fz.decompress(stream, ws=s["ws"])
    elif op == "roundtrip":
        out["field"] = fz.decompress(stream, header=s["header"], out=s["rec"], ws=s["ws"])
    return out


def _decoded(case, f):
    """The field a decompression gives back: each value times the 32-bit reciprocal of the bin
    width, rounded half away from zero in 32 bits (that is the stream's content), times the bin
    width in 64; 0 past the dims."""
    eb = _abs_bound(case, f)
    r = torch.tensor(1.0 / (eb * 2), dtype=torch.float32, device=f.device)
    v = f * r
    q = torch.trunc(v.double() + torch.copysign(torch.tensor(0.5, dtype=torch.float64, device=f.device), v.double()))
    q[case["x"] * case["y"] * case["z"]:] = 0
    return q * (eb * 2)


def exact(case, seed):
    if case["op"] == "batch":
        return {"streams": [None] * case["count"],
                "fields": [_decoded(m, _field(m, seed * 1000 + i)) for i, m in enumerate(_members(case))]}
    if case["op"] in ("compress", "compress-size"):
        return None
    field = _decoded(case, _field(case, seed))
    if case["op"] == "decompress":
        return {"field": field}
    if case["op"] == "stages":
        return dict.fromkeys(("codes", "shuffled", "bits", "flags", "sums", "chunks", "nnz"), None) | {"field": field}
    if case["op"] == "roundtrip":
        return {"stream": None, "field": field}
    return {"stream": None, "size": None, "field": field.cpu().numpy() if case["op"] == "host" else field}
