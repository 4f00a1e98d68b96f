"""Device FASTA ingest at the sizes where its kernels change their way: lines
around 32, 64 and 96 bytes, records of more than 32 and 256 lines, names longer
than a warp, files around the 4,096-byte tiles, and one '\\r' in a long record."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _record(rng, name_len, length, width, cr_at=None, tail=b"\n"):
    body = rng.choice(np.frombuffer(b"ACGTN", np.uint8), length).tobytes()
    lines = [body[i:i + width] for i in range(0, length, width)]
    if cr_at is not None and lines:
        lines[cr_at % len(lines)] += b"\r"
    name = (b"n" + b"0123456789" * (name_len // 10 + 1))[:name_len]
    return b">" + name + b" rest of the header\n" + b"\n".join(lines) + tail


@pytest.mark.parametrize("width", [1, 31, 32, 33, 64, 80, 95, 96, 97, 300])
@pytest.mark.parametrize("cr_at", [None, 0, 40])
def test_line_widths_and_counts(gpu_ctx, width, cr_at):
    rng = np.random.default_rng(width)
    data = b"".join(_record(rng, nl, lines * width + extra, width, cr_at, tail)
                    for nl, lines, extra, tail in
                    [(1, 1, 0, b"\n"), (31, 31, 0, b"\n"), (32, 32, 0, b"\n\n"),
                     (33, 33, width // 2, b"\n"), (64, 256, 0, b"\n"), (65, 257, 0, b"\n\n\n"),
                     (200, 700, width // 3, b"")])
    for cut in (len(data), len(data) - 1, len(data) - len(data) % 4096, 4097, 4096, 4095):
        part = data[:cut]
        want = oracle.parse_fasta_restated(part, min_contig=257, min_small=33)
        got = gpu_ctx.parse_fasta(part, 257, 33)
        assert got["num_seqs"] == want["num_seqs"]
        for kind in ("large", "small"):
            seqcat, offs, names = got[kind]
            assert [(names[i], seqcat[offs[i]:offs[i + 1]])
                    for i in range(len(names))] == want[kind]
