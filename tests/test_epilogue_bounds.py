"""The plain epilogues of a tile (write_pieces, csrc/gemm_tc.cu): a thread whose rows lie past the product's last row, or that has no column, is handed pointers
that are of no row - a bias one value short of a whole piece, for one - and must not read through any of them.  Checked in the source, since a run shows only what one
compiler made of it."""
import os
import re

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dynet_b200", "csrc", "gemm_tc.cu")


def test_threads_without_columns_read_nothing():
    text = re.sub(r"//[^\n]*", "", open(SOURCE).read())
    (body,) = re.findall(r"void write_pieces\([^)]*\)\s*\{(.*?)\n\}", text, re.S)
    leaves = re.search(r"if \(c >= c_hi\) return;", body)
    reads = re.search(r"\bat\(\w+\)", body)
    assert reads and leaves and leaves.start() < reads.start()
