"""The edge-list reader's two line parsers (plain "u v" lines by a branch-free
pass, others by the full rules): kinds of lines on either side of the line
between them, at the edges of blocks, against the CPU restatement.  Exact."""
import numpy as np
import pytest

import igraph_b200 as ig
from test_gpu_edgelist import expect, got, same

pytestmark = pytest.mark.gpu

KINDS = [b"1 2", b"123456789 7", b"1234567890 7", b"7 1234567890", b"7 4294967294", b"7\t8", b"7  8", b" 7 8", b"7 8 ",
         b"7 8\r", b"+7 8", b"007 08", b"", b"#7 8", b"999999999 999999999", b"0000000000 1", b"7 \xc2\xa08"]
BAD = [b"7", b"7 8 9", b"7 8x", b"7 x8", b"x 8", b"7 4294967296", b"42949672960 1", b"- 1", b"7 -1", b"7/8", b"7:8"]


@pytest.mark.parametrize("pad", [b"3 4", b"#" + b"c" * 45, b"#" + b"c" * 60, b"123456 654321"])
@pytest.mark.parametrize("at", [0, 254, 255, 256, 257, 511, 512, 700])
@pytest.mark.parametrize("end", [b"", b"\n"])
def test_line_kinds_at_block_edges(cuda_ok, pad, at, end):
    lines = [pad] * 720
    for i, k in enumerate(KINDS[:2] if at == 0 else KINDS):
        lines[at + i if at + i < 720 else i] = k
    text = b"\n".join(lines) + end
    assert same(expect(text), got(text))


@pytest.mark.parametrize("bad", BAD)
@pytest.mark.parametrize("at", [0, 255, 256, 600])
@pytest.mark.parametrize("long", [0, 12_000, 40_000])
def test_first_error(cuda_ok, bad, at, long):
    lines = [b"5 6"] * 640
    lines[40] = b"#" + b"l" * long
    lines[at] = bad
    lines[620] = b"later bad"
    text = b"\n".join(lines)
    assert same(expect(text), got(text))
