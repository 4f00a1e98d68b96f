"""The device's BGZF decoder on well-formed BAM files: members of every zlib level and
strategy, stored members and members of several deflate blocks, matches of all
lengths up to 258 and of distances below and above 32 bytes that overlap themselves;
against the host route (zlib), sums and means bit for bit."""
import struct
import zlib

import numpy as np
import pytest

from rabbitbin_b200.synth import bam_records, make_bam

pytestmark = pytest.mark.gpu
STRATEGIES = [zlib.Z_DEFAULT_STRATEGY, zlib.Z_FILTERED, zlib.Z_HUFFMAN_ONLY, zlib.Z_RLE, zlib.Z_FIXED]


def _member(data, comp):
    assert len(comp) + 26 <= 65536
    return (b"\x1f\x8b\x08\x04\0\0\0\0\0\xff\x06\0BC\x02\0" + struct.pack("<H", len(comp) + 25) + comp +
            struct.pack("<II", zlib.crc32(data), len(data)))


def _deflate(data, level, strategy, flushes=0, wbits=-15, mem=8):
    c = zlib.compressobj(level, zlib.DEFLATED, wbits, mem, strategy)
    out, step = b"", max(1, len(data) // (flushes + 1))
    for i in range(flushes):
        out += c.compress(data[i * step:(i + 1) * step])
        out += c.flush(zlib.Z_SYNC_FLUSH if i % 2 else zlib.Z_FULL_FLUSH)
    return out + c.compress(data[flushes * step:]) + c.flush()


def _split(records):
    out, o = [], 0
    while o < len(records):
        n = struct.unpack_from("<I", records, o)[0] + 4
        out.append(records[o:o + n])
        o += n
    return out


def _bam(names_lens, records, comp, size):
    """A BAM whose members hold whole records (about `size` bytes each); comp(i, data)
    the deflate stream of member i."""
    text = b"@HD\tVN:1.6\tSO:coordinate\n"
    head = b"BAM\1" + struct.pack("<i", len(text)) + text + struct.pack("<i", len(names_lens))
    for nm, ln in names_lens:
        head += struct.pack("<i", len(nm) + 1) + nm + b"\0" + struct.pack("<i", ln)
    members, cur = [head], b""
    for r in records:
        if cur and len(cur) + len(r) > size:
            members.append(cur)
            cur = b""
        cur += r
    members.append(cur)
    body = b"".join(_member(d, comp(i, d)) for i, d in enumerate(members) if d)
    return body + _member(b"", zlib.compress(b"")[2:-4])


def _check(gpu_ctx, bam, **kw):
    dev = gpu_ctx.bam_depth([bam], device_inflate=1, **kw)
    host = gpu_ctx.bam_depth([bam], device_inflate=0, **kw)
    assert dev["device_bams"] == 1 and dev["records"] == host["records"] > 0
    assert np.array_equal(dev["sums"], host["sums"]) and np.array_equal(dev["means"], host["means"])
    assert dev["sums"].sum() > 0


@pytest.fixture(scope="module")
def reads():
    lens = np.array([3000, 9000, 20000], np.uint32)
    bam = make_bam(lens, np.array([12.0, 9.0, 7.0]), seed=21)
    rec, tl, names = bam_records(bam)
    return [(n.encode(), int(ln)) for n, ln in zip(names, tl)], _split(rec)


@pytest.mark.parametrize("strategy", STRATEGIES)
@pytest.mark.parametrize("size", [300, 5000, 60000])
def test_levels_and_strategies(gpu_ctx, reads, strategy, size):
    """Level i of member i (0: stored blocks), flushes in every third one."""
    bam = _bam(*reads, lambda i, d: _deflate(d, i % 10, strategy, i % 3 if size > 300 else 0), size)
    _check(gpu_ctx, bam)


@pytest.mark.parametrize("wbits,mem", [(-9, 1), (-12, 5), (-15, 9)])
def test_windows_and_blocks(gpu_ctx, reads, wbits, mem):
    """Small windows, and with them many deflate blocks a member; also by 1 MB chunks."""
    bam = _bam(*reads, lambda i, d: _deflate(d, 9, zlib.Z_DEFAULT_STRATEGY, 0, wbits, mem), 50000)
    _check(gpu_ctx, bam)
    _check(gpu_ctx, bam, device_chunk_mb=1)


@pytest.mark.parametrize("period", [1, 2, 3, 5, 31, 32, 33, 64, 258, 300])
def test_self_overlapping_matches(gpu_ctx, period):
    """Records whose qualities repeat with a short period over thousands of bases."""
    rng = np.random.default_rng(period)
    unit = rng.integers(0, 60, period, dtype=np.uint8).tobytes()
    recs = []
    for k in range(60):
        n = 40 + int(rng.integers(0, 8000))
        seq = rng.integers(0, 256, (n + 1) // 2, dtype=np.uint8).tobytes()
        qual = (unit * (n // period + 1))[:n]
        name = b"r%d\0" % k
        core = struct.pack("<iiBBHHHiiii", 0, 10 + 5 * k, len(name), 60, 4680, 1, 0, n, -1, -1, 0)
        rec = core + name + struct.pack("<I", n << 4) + seq + qual + b"NMC\0"
        recs.append(struct.pack("<I", len(rec)) + rec)
    _check(gpu_ctx, _bam([(b"c0", 30000), (b"c1", 500)], recs,
                         lambda i, d: _deflate(d, (1, 6, 9)[i % 3], zlib.Z_DEFAULT_STRATEGY), 60000))
