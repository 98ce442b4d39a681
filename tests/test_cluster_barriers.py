"""A CTA may touch the shared memory of another CTA of its cluster only once that one is known to run: in every kernel that does, a wait on
the cluster's barrier comes before the first remote access.  Checked in the source, since a run does not show it."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dynet_b200", "csrc")
REMOTE = re.compile(r"\b(?:st|ld|red|atom)(?:\.async)?[\w.:]*\.shared::cluster|\bsend4\(|\bsend_bulk\(")
WAIT = re.compile(r"barrier\.cluster\.wait|\bcluster_wait\(\)|\bcluster_sync_all\(\)")


def kernels(text):
    """(name, body) of every __global__ function."""
    for m in re.finditer(r"__global__[^;{]*?(\w+)\s*\((?:[^(){}]|\([^()]*\))*\)\s*\{", re.sub(r"__launch_bounds__\([^)]*\)|__cluster_dims__\([^)]*\)", "", text)):
        text_ = m.string
        depth, k = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text_[k], 0)
            k += 1
        yield m.group(1), text_[m.end():k]


FOUND = [(os.path.basename(f), name, body) for f in sorted(glob.glob(os.path.join(CSRC, "*.cu")))
         for name, body in kernels(re.sub(r"//[^\n]*", "", open(f).read())) if REMOTE.search(body)]


def test_finds_the_kernels_that_talk_across_a_cluster():
    assert {n for _, n, _ in FOUND} >= {"k_lstm_seq_fwd", "k_lstm_rec_fwd", "k_lstm_rec_bwd", "k_rec_tc_fwd", "k_rec_tc_bwd", "k_col_cluster", "k_gemm_tc"}


@pytest.mark.parametrize("where,name,body", FOUND, ids=["%s:%s" % f[:2] for f in FOUND])
def test_waits_for_the_cluster_before_the_first_remote_access(where, name, body):
    wait = WAIT.search(body)
    assert wait and wait.start() < REMOTE.search(body).start()


def test_wide_backward_sends_only_behind_the_counter():
    """The exchange buffer of another CTA of the cluster is that CTA's scratch for row sums until it has published them, so every rank - one whose share of the
    reduction is empty included - waits for its column block's counter (go[cb]) before the partial sums of a product go out."""
    (body,) = [b for _, n, b in FOUND if n == "k_bwd_wide"]
    send = body.index("send4(")
    conditions = re.findall(r"if \(([^;{}]*)mbar_wait\(&go\[cb\], it & 1\b", body[:send])
    assert conditions == ["REC && ok && !"]
