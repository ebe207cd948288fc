"""The codec's work as its users run it, one case per call pattern, with the
real range of sizes, targets and outputs. Every case goes through the library's
public entry points (the C ABI of include/vc.h and include/vcg.h, by way of the
in-tree binding). Volumes are the benchmark's seeded synthetic scroll sheets.

Everything the codec returns is bytes or whole numbers, exact by definition, so
there is no 64-bit reference to compare with: exact() has no values."""
import ctypes
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "volume-compressor_gb300"))
import vc_gb300 as vc  # noqa: E402

LIBC = ctypes.CDLL(None)
LIBC.free.argtypes = [ctypes.c_void_p]

# LOD0 base_q that rate control picks for the synthetic volume at each target
Q0 = {10: 1.3139, 20: 2.5577, 50: 6.5357, 100: 13.558}
TARGETS = sorted(Q0)


def _case(name, kind, nx, ny, nz, target, **more):
    return dict({"name": name, "kind": kind, "nx": nx, "ny": ny, "nz": nz, "target": target}, **more)


def _drawn(kind, nx, ny, nz, target, **more):
    c = _case("", kind, nx, ny, nz, target, **more)
    del c["name"]
    return c


def listed():
    return [
        # random access to one 32^3 atom of a resident archive (a viewer's probe): the smallest call
        _case("atom_t20", "atom", 512, 512, 512, 20, lod=0),
        # a small unaligned box of a coarser LOD into host memory: ordinary interactive read
        _case("region_70x45x90_lod1", "region", 512, 512, 512, 20, lod=1, ex=70, ey=45, ez=90, device=False),
        # a training-crop sized unaligned box: some hundreds of atoms, none of its edges on an atom's
        _case("region_250x231x256", "region", 512, 512, 512, 20, lod=0, ex=250, ey=231, ez=256, device=False),
        # the smallest benchmark volume, whole LOD0 into host memory
        _case("lod0_256_t10_host", "lod", 256, 256, 256, 10, lod=0, device=False),
        # the headline: whole LOD0 of 1024^3, archive and output on the device
        _case("lod0_1024_t10", "lod", 1024, 1024, 1024, 10, lod=0, device=True),
        # the same volume at the strongest compression in use
        _case("lod0_1024_t100", "lod", 1024, 1024, 1024, 100, lod=0, device=True),
        # odd dims in every axis, middle compression: cut atoms along each far face
        _case("lod0_911x701x523_t50", "lod", 911, 701, 523, 50, lod=0, device=True),
        # open + decode + close of an archive in host memory, pageable output: a converter's loop
        _case("open_decode_512_t20", "open", 512, 512, 512, 20, lod=0),
        # many uneven boxes of any LOD in one call, outputs on the device: a data loader's batch
        _case("batch_600_boxes", "batch", 1024, 1024, 768, 20, boxes=600),
        # ingest with rate control from host memory, ragged dims
        _case("encode_rate_300x257x190_t20", "encode_rate", 300, 257, 190, 20),
        # ingest of a large volume on the device at chosen q
        _case("encode_q_1024_t10", "encode_q", 1024, 1024, 1024, 10),
        # the transform alone, both directions, over a volume on the device
        _case("dct_1024x1024x512", "dct", 1024, 1024, 512, 10, form=vc.DCT_BUTTERFLY),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["atom", "region", "region", "lod", "lod", "open", "batch", "encode_rate", "encode_q", "dct"])
    t = rng.choice(TARGETS)
    if kind == "atom":
        n = _log(rng, 64, 512)
        return _drawn(kind, n, _log(rng, 64, 512), _log(rng, 64, 512), t, lod=rng.choice([0, 1]))
    if kind == "region":
        lod = rng.choice([0, 0, 1, 2])
        d = [_log(rng, 300, 700) for _ in range(3)]
        e = [_log(rng, 20, min(256, (n >> lod) - 1)) for n in d]
        return _drawn(kind, *d, t, lod=lod, ex=e[0], ey=e[1], ez=e[2], device=rng.random() < 0.3)
    if kind == "lod":
        d = [_log(rng, 100, 1024) for _ in range(3)]
        return _drawn(kind, *d, t, lod=rng.choice([0, 0, 0, 1]), device=rng.random() < 0.7)
    if kind == "open":
        return _drawn(kind, *[_log(rng, 64, 512) for _ in range(3)], t, lod=0)
    if kind == "batch":
        return _drawn(kind, *[_log(rng, 300, 1000) for _ in range(3)], t, boxes=_log(rng, 16, 600))
    if kind == "encode_rate":
        return _drawn(kind, *[_log(rng, 33, 300) for _ in range(3)], t)
    if kind == "encode_q":
        return _drawn(kind, *[_log(rng, 64, 1024) for _ in range(3)], t)
    return _drawn(kind, *[32 * _log(rng, 1, 25) for _ in range(3)], t,
                      form=rng.choice([vc.DCT_BUTTERFLY, vc.DCT_IMMA]))


class _Dev:
    """A torch buffer where the binding takes a device buffer."""

    def __init__(self, nbytes, dtype=torch.uint8, n=None):
        self.t = torch.zeros(n if n is not None else nbytes, dtype=dtype, device="cuda")
        self.ptr, self.nbytes = self.t.data_ptr(), int(nbytes)


def _qs(target):
    q, out = Q0[target], []
    for _ in range(8):
        out.append(max(0.05, q))
        q *= 0.6
    return out


def _dims(c):
    return c["nx"], c["ny"], c["nz"]


def _lod_dims(d, lod):
    for _ in range(lod):
        d = tuple((n + 1) // 2 for n in d)
    return d


def _archive_bytes(c, seed):
    d = _dims(c)
    vol = vc.synth_device(*d, 0x5EED0000 + seed)
    s, data = vc.encode_q(vol, float(c["target"]), _qs(c["target"]), on_device=d)
    vol.free()
    if s:
        raise RuntimeError("encode failed (%d): %s" % (s, vc.last_error()))
    return data


def _box(rng, d, e):
    o = [rng.randint(0, n - k) for n, k in zip(d, e)]
    return tuple(o) + tuple(a + k for a, k in zip(o, e))


def prepare(case, seed):
    c, rng = dict(case), random.Random(seed)
    kind = c["kind"]
    if kind in ("atom", "region", "lod", "batch"):
        c["arc"] = vc.Archive(_archive_bytes(c, seed))
        if c["arc"].make_resident():
            raise RuntimeError(vc.last_error())
    if kind == "atom":
        c["at"] = [rng.randrange((n + 31) // 32) for n in _lod_dims(_dims(c), c["lod"])]
        c["out"] = np.zeros(32768, np.uint8)
    elif kind in ("region", "lod"):
        d = _lod_dims(_dims(c), c["lod"])
        e = (c["ex"], c["ey"], c["ez"]) if kind == "region" else d
        c["box"] = _box(rng, d, e)
        n = e[0] * e[1] * e[2]
        c["out"] = _Dev(n) if c["device"] else np.zeros(n, np.uint8)
    elif kind == "open":
        c["data"] = np.frombuffer(_archive_bytes(c, seed), np.uint8).copy()
        c["out"] = np.zeros(c["nx"] * c["ny"] * c["nz"], np.uint8)
    elif kind == "batch":
        reqs, size, shape = [], 0, random.Random(c["boxes"])
        for _ in range(c["boxes"]):   # the benchmark's batch: edges 32-256, LOD 0-3; the offsets are the seed's
            lod = shape.randrange(4)
            d = _lod_dims(_dims(c), lod)
            b = _box(rng, d, [min(n, shape.randint(32, 256)) for n in d])
            reqs.append((lod, b, size))
            size += (b[3] - b[0]) * (b[4] - b[1]) * (b[5] - b[2])
        c["out"] = _Dev(size)
        arr = (vc.RegionRequest * len(reqs))()
        for i, (lod, b, off) in enumerate(reqs):
            arr[i].lod, arr[i].box, arr[i].out = lod, vc.Box(*b), c["out"].ptr + off
        c["reqs"], c["status"] = arr, np.zeros(len(reqs), np.int32)
    elif kind in ("encode_rate", "encode_q", "dct"):
        c["vol"] = vc.synth_device(*_dims(c), 0x5EED0000 + seed)
        n = c["nx"] * c["ny"] * c["nz"]
        if kind == "encode_rate":
            c["host"] = c["vol"].download(n)
            c["vol"].free()
        if kind != "dct":   # the caller's archive buffer, and how much of it is filled
            c["out"], c["len"] = np.zeros(2 * n // c["target"] + (16 << 20), np.uint8), 0
        else:
            c["coef"], c["dc"] = _Dev(4 * n, torch.int32, n), _Dev(n // 32768)
            c["back"] = _Dev(n)
    torch.cuda.synchronize()
    return c


def _ok(s):
    if s:
        raise RuntimeError("status %d: %s" % (s, vc.last_error()))


def _encoded(c, call, *a):
    """An encode call of the C ABI, its malloc'ed archive taken over into the caller's buffer."""
    p, n = ctypes.c_void_p(), ctypes.c_size_t()
    _ok(call(*a, ctypes.byref(p), ctypes.byref(n)))
    if n.value > c["out"].size:
        raise RuntimeError("archive of %d bytes" % n.value)
    ctypes.memmove(c["out"].ctypes.data, p, n.value)
    LIBC.free(p)
    c["out"][n.value:c["len"]] = 0
    c["len"] = n.value
    return [c["out"], n.value]


def run(state):
    c = state
    kind = c["kind"]
    if kind == "atom":
        _ok(c["arc"].decode_atom(c["lod"], *c["at"], out=c["out"])[0])
        return c["out"]
    if kind == "region":
        if c["device"]:
            _ok(c["arc"].decode_region_device(c["lod"], c["box"], c["out"]))
            return c["out"].t
        _ok(c["arc"].decode_region(c["lod"], c["box"], out=c["out"])[0])
        return c["out"]
    if kind == "lod":
        if c["device"]:
            _ok(c["arc"].decode_lod_device(c["lod"], c["out"]))
            return c["out"].t
        _ok(c["arc"].decode_lod(c["lod"], out=c["out"])[0])
        return c["out"]
    if kind == "open":
        h = vc.lib().vc_open(c["data"].ctypes.data, c["data"].size)
        s = vc.lib().vc_decode_lod(h, 0, c["out"].ctypes.data, ctypes.byref(vc.Dims()))
        vc.lib().vc_close(h)
        _ok(s)
        return c["out"]
    if kind == "batch":
        _ok(vc.lib().vcg_decode_regions(c["arc"].h, len(c["reqs"]), c["reqs"], 1, c["status"].ctypes.data))
        return [c["out"].t, c["status"]]
    if kind == "encode_rate":
        return _encoded(c, vc.lib().vc_encode, c["host"].ctypes.data, vc.Dims(*_dims(c)), ctypes.c_float(c["target"]))
    if kind == "encode_q":
        q = (ctypes.c_float * 8)(*_qs(c["target"]))
        return _encoded(c, vc.lib().vcg_encode_q, c["vol"].ptr, 1, vc.Dims(*_dims(c)), ctypes.c_float(c["target"]), q)
    s, r0 = vc.dct_forward(c["vol"], _dims(c), vc.DCT_ATOM_DC, c["form"], c["coef"], c["dc"])
    _ok(s)
    s, r1 = vc.dct_inverse(c["coef"], _dims(c), vc.DCT_ATOM_DC, c["form"], c["back"], c["dc"])
    _ok(s)
    return [c["coef"].t, c["dc"].t, c["back"].t, r0, r1]


def work(case):
    """Payload and voxel bytes, each once; the multiply-adds of the three
    32-point butterfly passes (344 multiplies a line). The coder's serial
    decisions are neither."""
    c, kind = case, case["kind"]
    d = _dims(c)
    n = d[0] * d[1] * d[2]
    if kind == "atom":
        n = 32768
    elif kind == "region":
        n = c["ex"] * c["ey"] * c["ez"]
    elif kind == "lod":
        e = _lod_dims(d, c["lod"])
        n = e[0] * e[1] * e[2]
    elif kind == "batch":
        n = c["boxes"] * 144 ** 3   # mean box
    if kind == "dct":
        return {"bytes": 2.0 * (n + 4 * n), "flops": 2.0 * n * 64.5}
    pyr = 8 / 7 if kind.startswith("encode") else 1.0
    return {"bytes": pyr * n * (1 + 1 / c["target"]), "flops": pyr * n * 64.5}


def exact(case, seed):
    return None
