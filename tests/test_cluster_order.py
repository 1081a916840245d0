"""What the kernels' sources must order around a thread-block cluster, read from the sources: a missing wait there shows
on a GPU only by chance."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rwkvstic_b200", "csrc")
REMOTE = ("map_shared_rank(", "leader_addr(", "mbar_arrive_leader(")          # another CTA's shared memory
BARRIER = ("cluster_sync();", "cluster.sync();", "cluster.barrier_wait(")


def closing(text, at, pair):
    """Index behind the bracket that closes the one in front of `at`."""
    depth = 1
    while depth:
        depth += {pair[0]: 1, pair[1]: -1}.get(text[at], 0)
        at += 1
    return at


def kernels():
    """(file, name, body without comments) of every __global__ function."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)
        for m in re.finditer(r"__global__\s+void\s+", text):
            at = m.end()
            if text.startswith("__launch_bounds__(", at):
                at = closing(text, at + len("__launch_bounds__("), "()")
            head = re.compile(r"\s*(\w+)\s*\(").match(text, at)
            start = text.index("{", closing(text, head.end(), "()")) + 1
            yield os.path.basename(path), head.group(1), text[start:closing(text, start, "{}")]


CLUSTERED = [pytest.param(body, id=f"{f}:{name}") for f, name, body in kernels() if any(t in body for t in REMOTE)]


def test_the_clustered_kernels_are_found():
    ids = " ".join(p.id for p in CLUSTERED)
    assert all(k in ids for k in ("tile_gemm_kernel", "dense_tile_gemm_kernel", "sample_typical_kernel")), ids


@pytest.mark.parametrize("body", CLUSTERED)
def test_a_cluster_barrier_comes_before_the_first_access_to_another_ctas_memory(body):
    """A CTA of a cluster may start after its peers: its shared memory exists for them once a barrier has been met."""
    first = min(body.find(t) for t in REMOTE if t in body)
    assert any(-1 < body.find(t) < first for t in BARRIER)


@pytest.mark.parametrize("body", [pytest.param(body, id=f"{f}:{name}") for f, name, body in kernels() if "umma_commit<kPair>(" in body])
def test_a_producer_waits_for_the_commits_that_arrive_in_its_cta(body):
    """tcgen05.commit with multicast arrives on a barrier in both CTAs of a pair.  A CTA that leaves while such an
    arrival is on its way has it land in shared memory that is no longer its own, so the producer waits for the
    release of every stage after its last copy and before the barrier in front of the exit."""
    last_copy = max(m.start() for m in re.finditer(r"&Sg\.xmap", body))
    assert last_copy < body.find("ring_drain(empty0") < body.rfind("cluster_sync();")
