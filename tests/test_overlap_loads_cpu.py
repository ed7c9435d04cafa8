"""A kernel launched to overlap its predecessor exists while that one still
writes, so what kernels write must not be read through the read-only path
there: no read-only load in the files whose kernels are launched so, and
read-only (const __restrict__) parameters only for the work lists, which no
kernel writes.  Read from the source: a stale read cannot be brought about."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "su2dmrg_gb300", "csrc")
LISTS = {"GemmTile", "GemmSeg", "PackJob", "int2", "OzTile", "OzSeg", "RedTile"}


def test_overlapped_kernels_read_data_by_plain_loads():
    files = 0
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith(".cu"):
            continue
        with open(os.path.join(CSRC, name)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        if "wait_for_predecessor()" not in text:
            continue
        files += 1
        assert "__ldg(" not in text and "ld.global.nc" not in text and "__ldcs(" not in text, name
        for m in re.finditer(r"__global__\s+void[^;{]*?\w+\s*\(([^{};]*)\)\s*\{", text):
            body = text[m.end(): text.index("\n}", m.end())]
            if "wait_for_predecessor()" in body:
                read_only = set(re.findall(r"const\s+(\w+)\s*\*\s*__restrict__", m.group(1)))
                assert read_only <= LISTS, (name, read_only)
    assert files == 3
