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


def _launched_early():
    """The kernels that files hand to launch_early, by name or through a variable."""
    names = set()
    for name, text in _files():
        for m in re.finditer(r"(?<!void )\blaunch_early(_clusters)?\(", text):
            args = text[m.end():_closing(text, m.end() - 1, "()")]
            kern = args.split(",")[1 if m.group(1) else 0].strip()
            if kern == "kern" and name == "common.cuh":
                continue
            direct = re.match(r"\w+_kernel\b", kern)
            if direct:
                names.add(direct.group(0))
                continue
            variable = re.match(r"\w+", kern).group(0)              # every kernel that it is given in this file
            given = "".join(re.findall(r"\b%s\b[^;=]*=([^;]*);" % variable, text))
            if not given:                                           # the parameter of a local launcher
                given = "".join(re.findall(r"\blaunch\(([^;]*);", text))
            found = re.findall(r"\w+_kernel\b", given)
            assert found, (name, kern)
            names.update(found)
    return sorted(names)


@pytest.mark.parametrize("kernel", _launched_early())
def test_kernels_launched_early_wait_before_they_touch_memory(kernel):
    params, body = KERNELS[kernel][1:]
    assert "wait_previous();" in body, "never waits"
    before, after = body.split("wait_previous();", 1)
    structs = re.findall(r"const \w+ (p|pg)\b", params)
    for p in re.findall(r"\*\s*(?:__restrict__\s*)?(\w+)", params):
        assert not re.search(r"\b%s\b" % p, before), f"{p} is used before the wait"
    for p in structs:                                                # sizes may be read; what their pointers lead to may not
        assert not re.search(r"\b%s\.\w+\[" % p, before), f"an array of {p} is read before the wait"


@pytest.mark.parametrize("kernel", [k for k, (_, _, body) in KERNELS.items() if "wait_previous();" in body])
def test_arguments_taken_for_constant_are_taken_anew_behind_the_wait(kernel):
    """Loads through a const __restrict__ argument may be moved ahead of the wait: the pointer goes through after_wait."""
    params, body = KERNELS[kernel][1:]
    for p in re.findall(r"const [^,]*?\*\s*__restrict__\s*(\w+)", params):
        assert re.search(r"\b%s = after_wait\(%s\);" % (p, p), body.split("wait_previous();", 1)[1]), f"{p} is not"


@pytest.mark.parametrize("kernel", [k for k, (_, _, body) in KERNELS.items() if "wait_previous();" in body])
def test_no_non_coherent_loads_in_kernels_launched_early(kernel):
    """They ask that nobody writes the memory for as long as the kernel lives, which begins while the kernel ahead still writes."""
    assert not re.search(r"ld_vec8_stream|__ldg|ld\.global\.nc", KERNELS[kernel][2])
