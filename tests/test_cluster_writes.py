"""A block of a thread-block cluster may write into a peer's shared memory only once the peer runs: in every kernel that does,
the first such write stands after a wait at the cluster's barrier.  Read off the source; no GPU is needed."""
import os
import re

import pytest

import rocml_b200

CSRC = os.path.join(os.path.dirname(rocml_b200.__file__), "csrc")
WRITE = re.compile(r"\b(st_cluster|st_cluster_f32|mbar_arrive_cluster|tma_load_2d_pair|mma_commit_pair)\s*\(|shared::cluster\.(f32|u32|b32)\s*\[%0\]")
WAIT = re.compile(r"\b(cluster_wait|cluster_wait_acquire|cluster_sync_all)\s*\(")


def kernels(path):
    """(name, body) of every __global__ function of a file, comments taken out."""
    with open(path) as f:
        text = re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)
    for m in re.finditer(r"__global__", text):
        at = text.index("{", m.end())
        name = re.findall(r"(\w+)\s*\(", text[m.end():at])[-1]
        depth, end = 0, at
        while True:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
            if depth == 0:
                break
        yield name, text[at:end]


def writers():
    out = []
    for f in sorted(os.listdir(CSRC)):
        if f.endswith(".cu"):
            out += [pytest.param(body, id=f"{f}:{name}") for name, body in kernels(os.path.join(CSRC, f)) if WRITE.search(body)]
    return out


def test_the_writers_are_found():
    names = {p.id.split(":")[1] for p in writers()}
    assert {"gemm_tcgen05_kernel", "gemm_tcgen05_pair_kernel", "attention_decode_kernel"} <= names


@pytest.mark.parametrize("body", writers())
def test_a_peer_is_known_to_run_before_it_is_written_to(body):
    wait = WAIT.search(body)
    assert wait is not None and wait.start() < WRITE.search(body).start()
