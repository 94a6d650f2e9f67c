"""CTAs of a cluster leave together: in every kernel that writes to or reads from another
CTA's shared memory, or signals its barriers, a cluster-wide barrier follows the last such
access, also on the way of a wait that ran out (an access to the shared memory of a CTA that
has left is a fault).  Read from the source: the failure needs a hung wait."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "deep-learning_b200", "csrc")
REMOTE = re.compile(r"st_cluster4\(|st_cluster_int\(|mbar_arrive_cluster\(|umma_pair_commit\(|send_block\(|"
                    r"ld\.shared::cluster|tma_pair_\dd\(|load_plane<|\.send\(|\.send2\(|send_cell\(")
TOGETHER = re.compile(r"cluster_sync_all\(\)|cluster_wait\(\)|\.finish\(\)")


def body(name, function):
    """Text of `function` in source `name`, comments taken out."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    at = re.search(r"\bvoid\b[^;{}]*\b" + function + r"\(", text)
    start = text.index("{\n", at.end())
    depth, end = 0, start
    for end in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        if depth == 0:
            break
    return text[start:end]


@pytest.mark.parametrize("name,function", [
    ("gemm_pair.cu", "gemm_x3_pair_kernel"), ("gemm_mid.cu", "gemm_mid_kernel"), ("gemm_direct.cu", "gemm_direct_kernel"),
    ("gemm_small.cu", "gemm_small_kernel"), ("planes.cu", "split_column_lines"),
    ("lstm_walk.cu", "lstm_forward_walk_kernel"), ("lstm_walk.cu", "lstm_backward_walk_kernel")])
def test_barrier_after_the_last_remote_access(name, function):
    text = body(name, function)
    last = [m.end() for m in REMOTE.finditer(text)]
    assert last, "no access to another CTA found"
    assert any(m.start() > max(last) for m in TOGETHER.finditer(text))


def test_no_other_kernel_reaches_into_a_cluster():
    # tc_*.cuh: the wrappers; gemm_tcgen05.cu: TMA loads into its own shared memory.
    known = {"gemm_pair.cu", "gemm_mid.cu", "gemm_direct.cu", "gemm_small.cu", "planes.cu", "lstm_walk.cu", "tc_ptx.cuh",
             "tc_pair.cuh"}
    for name in sorted(set(os.listdir(CSRC)) - known):
        assert not re.search(r"map_to_cta|mapa\.|shared::cluster", open(os.path.join(CSRC, name)).read()), name
