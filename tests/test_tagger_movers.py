"""What the tagger's benchmark counts for the four movers of a pass is what the driver (host/tagger.cc) moves: every one a copy, a read and a write per value."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _read(*path):
    return open(os.path.join(ROOT, *path)).read()


def test_the_benchmark_counts_the_calls_that_are_made():
    driver = re.sub(r"//[^\n]*", "", _read("dynet_b200", "host", "tagger.cc"))
    movers = re.findall(r"for \(int dr = 0; dr < 2; \+\+dr\) \{\s*if \(m\.time_movers\)[^;]*;\s*gpu::(\w+)\(", driver)
    assert movers == ["parallel_memcpy", "parallel_memcpy"] and "parallel_accumulate" not in driver
    bench = _read("bench.py")
    assert re.search(r"^TAGGER_MOVERS = 4\b", bench, re.M) and "algo = TAGGER_MOVERS * 2 * slice_bytes" in bench
    assert "k_ragged_accumulate" not in bench and "k_ragged_probe" not in bench
