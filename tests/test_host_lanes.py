"""The per-lane range decoder in the loop its kernels run (RcLane::rounds, with
no zeros at once and with six) built for the host (tests/host_lanes.cpp): the
oracle's status and levels, an end and no load of a word outside the stream, on crafted streams whose escape prefix is
longer than any level needs at every distance from the ends of the band and of
the stream, on runs of 0xFF, on coded noise, cut and random streams. No GPU needed."""
import os
import struct
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from rcstream import RangeEncoder
from test_host_decoders import SANITIZE, expected, other_streams


def build(tmp_path_factory, flags, name):
    exe = str(tmp_path_factory.mktemp(name) / name)
    src = os.path.join(ROOT, "tests", "host_lanes.cpp")
    inc = os.path.join(ROOT, "volume-compressor_gb300", "csrc")
    r = subprocess.run(["g++", *flags, "-std=c++17", "-w", "-I", inc, src, "-o", exe], capture_output=True, text=True)
    return exe, r


@pytest.fixture(scope="module", params=["plain", "sanitized"])
def harness(tmp_path_factory, request):
    if request.param == "plain":
        exe, r = build(tmp_path_factory, ["-O2"], "host_lanes")
        if r.returncode:
            pytest.fail(r.stderr[-2000:])
        return exe
    exe, r = build(tmp_path_factory, SANITIZE, "host_lanes_san")
    if r.returncode:
        pytest.skip("no AddressSanitizer / UBSan with this compiler: " + r.stderr[-200:])
    return exe


def crafted(eob, levels, ones, tail):
    """Coder bytes: `levels` (magnitudes, 0 for a zero) at scan positions 0, 1,
    ..., then one that escapes with a prefix of `ones` ones, then `tail` bytes."""
    e = RangeEncoder()
    sig, mag = [2048], [2048] * 12   # band 0 has 364 positions
    for i in range(15, -1, -1):
        e.bypass((eob >> i) & 1)
    for m in levels:
        e.bit(sig, 0, int(m != 0))
        if m:
            for k in range(12):
                e.bit(mag, k, int(m > k + 1))
                if m <= k + 1:
                    break
            if m > 12:
                x = m - 11
                nb = x.bit_length() - 1
                for _ in range(nb):
                    e.bypass(1)
                e.bypass(0)
                for b in range(nb - 1, -1, -1):
                    e.bypass((x >> b) & 1)
            e.bypass(m & 1)
    e.bit(sig, 0, 1)
    for k in range(12):
        e.bit(mag, k, 1)
    for _ in range(ones):
        e.bypass(1)
    return e.finish() + bytes(tail)


def overlong_streams():
    rng = np.random.default_rng(0x33)
    out = []
    for eob in (1, 5, 12, 200, 4000, 30000):
        for before in (0, 1, 2, 3, 4, 5, 6, 7, 8, 13, 40):
            if before >= eob:
                continue
            for ones in (32, 33, 34, 40):
                for tail in (0, 1, 3, 7, 15, 16, 17, 18, 30, 61, 200):
                    levels = rng.choice([0, 0, 1, 2, 5, 14, 3000], before)
                    out.append(crafted(eob, [int(m) for m in levels], ones, rng.integers(0, 256, tail).astype(np.uint8)))
    for n in list(range(0, 80)) + [200, 4096]:
        out.append(b"\xff" * n)
        out.append(b"\0" + b"\xff" * n)
    return out


def run(harness, oracle, streams, tmp_path, *more):
    path = str(tmp_path / "streams.bin")
    with open(path, "wb") as f:
        f.write(struct.pack("<I", len(streams)))
        for s in streams:
            bad, ent = expected(oracle, s)
            f.write(struct.pack("<III", len(s), bad, len(ent)))
            f.write(s)
            f.write(ent.astype("<u4").tobytes())
    r = subprocess.run([harness, path, *more], capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stderr[-3000:]
    return {name: (int(diff), int(endless), int(outside)) for name, diff, endless, outside, _ in
            (line.split() for line in r.stdout.strip().splitlines())}


def test_overlong_prefix_ends(harness, oracle, tmp_path):
    streams = overlong_streams()
    bad = [expected(oracle, s)[0] for s in streams]
    assert sum(bad) > len(streams) // 3 and sum(bad) < len(streams)
    assert run(harness, oracle, streams, tmp_path) == {"dense": (0, 0, 0), "zeros": (0, 0, 0)}


def test_noise_cut_and_random_streams(harness, oracle, tmp_path):
    assert run(harness, oracle, other_streams(oracle), tmp_path) == {"dense": (0, 0, 0), "zeros": (0, 0, 0)}


@pytest.mark.parametrize("more", ["0x7FFFFFFF", "0x80000064", "0xFFF00000"])
def test_length_past_two_gigabytes(harness, oracle, tmp_path, more):
    """A payload may claim up to 4 GiB; the decoder takes what its levels need."""
    assert run(harness, oracle, other_streams(oracle), tmp_path, more) == {"dense": (0, 0, 0), "zeros": (0, 0, 0)}
