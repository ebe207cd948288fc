"""The coder with an atom per lane (csrc/rc_encode.cuh, rounds over carry-free
sums) built for the host (tests/host_enc_lanes.cpp) and checked against the
oracle's level encoder: the bytes its sums stand for on golden atoms' levels and
on random lists, the count alone where a list has more sums than a slot, on both
sides of that line. No GPU needed."""
import os
import struct
import subprocess

import numpy as np
import pytest

from conftest import ROOT, load_archive
from test_host_encoder import SCAN, entries

SLOT_MAX = 32768 - 512 + 5   # bytes from which a list has too many sums (kSumsMax + 5)


@pytest.fixture(scope="module", params=["plain", "sanitized"])
def harness(tmp_path_factory, request):
    flags = {"plain": ["-O2"], "sanitized": ["-O1", "-g", "-fsanitize=address,undefined", "-fno-omit-frame-pointer",
                                             "-fno-sanitize-recover=undefined"]}[request.param]
    exe = str(tmp_path_factory.mktemp("enc_lanes") / "enc_lanes")
    r = subprocess.run(["g++", *flags, "-std=c++17", "-w", "-I", os.path.join(ROOT, "volume-compressor_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "host_enc_lanes.cpp"), "-o", exe], capture_output=True, text=True)
    if r.returncode and request.param == "sanitized":
        pytest.skip("no AddressSanitizer / UBSan with this compiler: " + r.stderr[-200:])
    assert r.returncode == 0, r.stderr[-2000:]
    return exe


def coded(oracle, lv):
    lv = np.ascontiguousarray(lv, np.int16)
    buf = np.zeros(200000, np.uint8)
    n = oracle.lib().orc_enc_levels(lv.ctypes.data, buf.ctypes.data, len(buf))
    assert n > 0
    return buf[:n].tobytes()


def run(harness, oracle, rasters, tmp_path):
    path = str(tmp_path / "lists.bin")
    with open(path, "wb") as f:
        f.write(struct.pack("<I", len(rasters)))
        for lv in rasters:
            e, b = entries(lv), coded(oracle, lv)
            f.write(struct.pack("<II", len(e), len(b)))
            f.write(e.astype("<u4").tobytes())
            f.write(b)
    r = subprocess.run([harness, path], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    diff, past, n = map(int, r.stdout.split())
    assert n == len(rasters)
    return diff, past


def test_golden_atom_levels(harness, oracle, golden, tmp_path):
    rasters = []
    for name in ("synth_64_t10", "synth_flat_96x64x33_t100", "ref_test_basic", "extreme_sat", "extreme_voxel"):
        data = load_archive(golden[name])
        a = oracle.Archive(data)
        for lod in range(a.nlod):
            _, (nx, ny, nz) = a.lod_dims(lod)
            for az in range((nz + 31) // 32):
                for ay in range((ny + 31) // 32):
                    for ax in range((nx + 31) // 32):
                        _, off, ln = a.payload_range(lod, az, ay, ax)
                        if ln <= 1:
                            continue
                        st = data[off + 1:off + ln]
                        lv = np.zeros(32768, np.int16)
                        buf = np.frombuffer(st + b"\0" * 8, np.uint8)
                        assert oracle.lib().orc_dec_levels(buf.ctypes.data, len(st), lv.ctypes.data) == 0
                        rasters.append(lv)
        a.close()
    assert len(rasters) > 100
    assert run(harness, oracle, rasters, tmp_path) == (0, 0)


def test_random_level_lists(harness, oracle, tmp_path):
    rng = np.random.default_rng(0xE7D)
    rasters = [np.zeros(32768, np.int16), np.full(32768, 32767, np.int16)]   # empty; every position at the clamp
    rasters += [rng.integers(-m, m + 1, 32768).astype(np.int16) for m in (1, 3, 12, 13, 40)]   # dense
    for n in (1, 2, 3, 4, 5, 31, 32, 33, 400):   # sparse, any magnitude
        lv = np.zeros(32768, np.int16)
        pos = rng.choice(32768, n, replace=False)
        lv[pos] = (rng.integers(1, 32768, n) * rng.choice([-1, 1], n)).astype(np.int16)
        rasters.append(lv)
    for m in (1, 11, 12, 13, 14, 27, 28, 1000, 32767):   # one level, at the last scan position
        lv = np.zeros(32768, np.int16)
        lv[SCAN[-1]] = m
        rasters.append(lv)
    past = sum(len(coded(oracle, lv)) >= SLOT_MAX for lv in rasters)
    assert past >= 1
    assert run(harness, oracle, rasters, tmp_path) == (0, past)


def test_around_the_slot(harness, oracle, tmp_path):
    """Lists cut so that their bytes lie on both sides of a slot's sums."""
    rng = np.random.default_rng(0xE7E)
    full = rng.integers(-900, 901, 32768).astype(np.int16)
    lo, hi = 1, 32768   # scan positions kept: the most whose bytes fit
    while hi - lo > 1:
        mid = (lo + hi) // 2
        lv = full.copy()
        lv[SCAN[mid:]] = 0
        lo, hi = (mid, hi) if len(coded(oracle, lv)) < SLOT_MAX else (lo, mid)
    rasters = []
    for k in range(lo - 6, lo + 8):
        lv = full.copy()
        lv[SCAN[k:]] = 0
        rasters.append(lv)
    past = sum(len(coded(oracle, lv)) >= SLOT_MAX for lv in rasters)
    assert 0 < past < len(rasters)
    assert run(harness, oracle, rasters, tmp_path) == (0, past)
