"""The warp's branches of the DEFLATE decoder (table build by votes, paired literal
stores, matches stored at the next one, 8-byte refills) on 32 lanes that take turns
on the host, under AddressSanitizer: well-formed streams of every kind decode to
zlib's bytes, damaged ones end with the one-lane decoder's status, and nothing is
read or written out of bounds."""
import os
import subprocess
import zlib

import numpy as np
import pytest

from test_inflate_cpu import _deflate, _payloads, _run, dec  # noqa: F401

HERE = os.path.dirname(os.path.abspath(__file__))
STRATEGIES = [zlib.Z_DEFAULT_STRATEGY, zlib.Z_FILTERED, zlib.Z_HUFFMAN_ONLY, zlib.Z_RLE, zlib.Z_FIXED]


@pytest.fixture(scope="module")
def lanes(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("lanes")
    exe = str(tmp / "inflate_lanes")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=address",
                    "-fno-omit-frame-pointer", os.path.join(HERE, "native", "inflate_lanes.cpp"),
                    "-o", exe], check=True)

    def run(recs):
        path = tmp / "streams.bin"
        with open(path, "wb") as f:
            for blob, n in recs:
                f.write(len(blob).to_bytes(4, "little") + n.to_bytes(4, "little") + blob)
        r = subprocess.run([exe, str(path)], capture_output=True, text=True,
                           env=dict(os.environ, ASAN_OPTIONS="detect_leaks=0"))
        assert r.returncode == 0, r.stderr[-3000:]
        return tuple(map(int, r.stdout.split()))
    return run


def _matches():
    """Payloads of matches of every length and many distances, below and above the
    32 bytes a warp copies at once, each overlapping itself where it is longer than
    its distance."""
    rng = np.random.default_rng(8)
    out = {}
    for period in (1, 2, 3, 5, 7, 31, 32, 33, 64, 257, 258, 300, 4000):
        unit = rng.integers(0, 256, period, dtype=np.uint8).tobytes()
        body = bytearray()
        for k in range(40):
            n = 3 + int(rng.integers(0, 600))
            body += (unit * (n // period + 2))[:n]
            body += rng.integers(0, 256, int(rng.integers(0, 3)), dtype=np.uint8).tobytes()
        out[f"period{period}"] = bytes(body)[:16000]
    return out


def test_well_formed_streams(lanes, dec):  # noqa: F811
    recs = []
    for name, data in {**_payloads(), **_matches()}.items():
        data = data[:24000]
        for i, level in enumerate((0, 1, 6, 9)):
            comp = _deflate(data, level, STRATEGIES[(i + len(recs)) % 5])
            assert _run(dec, comp, len(data)) == (0, data), (name, level)
            recs.append((comp, len(data)))
    # many deflate blocks, a stored one among them
    p = _payloads()
    c = zlib.compressobj(6, zlib.DEFLATED, -15)
    parts = [p["text"][:9000], p["random"][:3000], p["bam"][:9000], b"", p["zeros"][:2000]]
    comp = b"".join(c.compress(x) + c.flush(zlib.Z_SYNC_FLUSH) for x in parts) + c.flush()
    recs.append((comp, sum(map(len, parts))))
    assert lanes(recs) == (len(recs), len(recs))


def test_damaged_streams(lanes):
    rng = np.random.default_rng(12)
    recs = []
    for name, data in {**_payloads(), **_matches()}.items():
        data = data[:5000]
        for level, st in ((1, zlib.Z_DEFAULT_STRATEGY), (9, zlib.Z_DEFAULT_STRATEGY), (6, zlib.Z_FIXED),
                          (0, zlib.Z_DEFAULT_STRATEGY)):
            comp = _deflate(data, level, st)
            for _ in range(4):
                bad = bytearray(comp)
                for _ in range(int(rng.integers(1, 4))):
                    if len(bad):
                        bad[int(rng.integers(0, len(bad)))] ^= 1 << int(rng.integers(0, 8))
                recs.append((bytes(bad), len(data)))
                recs.append((bytes(comp[:int(rng.integers(0, len(comp) + 1))]), len(data)))
                recs.append((bytes(bad), int(rng.integers(0, 6000))))
    runs, ok = lanes(recs)
    assert runs == len(recs) and ok < runs
