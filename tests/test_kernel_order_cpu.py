"""Rules of order that the kernels' sources keep and that a run on a GPU may pass by luck: what a kernel does before it may."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "swiftllm_b200", "csrc")


def _files():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, name)) as f:
                yield name, re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)


def _closing(text, at, pair):
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i
    raise AssertionError("unbalanced")


def _kernels():
    """name -> (file, parameters, body) of every __global__ function."""
    found = {}
    for name, text in _files():
        for m in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\s*\(", text):
            end = _closing(text, m.end() - 1, "()")
            begin = text.index("{", end)
            found[m.group(1)] = (name, text[m.end():end], text[begin:_closing(text, begin, "{}") + 1])
    return found


KERNELS = _kernels()
REMOTE = re.compile(r"map_shared_rank|ld_cluster\(|\bmapa\b")


@pytest.mark.parametrize("kernel", [k for k, (_, _, body) in KERNELS.items() if REMOTE.search(body)])
def test_other_ctas_have_started_before_their_shared_memory_is_touched(kernel):
    body = KERNELS[kernel][2]
    waits = [m.start() for m in re.finditer(r"\bcluster_sync_all\(|\bcluster\.(?:sync|barrier_wait)\(", body)]
    remote = [m.start() for m in REMOTE.finditer(body)]
    assert waits and waits[0] < remote[0] and waits[-1] > remote[0]           # started; and nobody leaves, or reads, too early
