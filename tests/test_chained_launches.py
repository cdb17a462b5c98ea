"""The rule of chained launches (csrc/launch.cuh) in the sources of the light-tree build and the sort, whose kernels
read what the kernel before them wrote: a kernel that waits for its predecessor reads nothing by the read-only path
(__ldg, const __restrict__ parameters), and waits before anything else."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "caelix-renderer_b200", "csrc")


def functions(source):
    """(name, parameters, body) of every device function and kernel."""
    for m in re.finditer(r"(?:__global__|__device__)[^;{}]*?(\w+)\s*\(([^;{}]*)\)\s*\{", source):
        depth, at = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(source[at], 0)
            at += 1
        name = re.findall(r"(\w+)\s*\(", m.group(0).replace("__launch_bounds__", ""))
        yield name, m.group(0), source[m.end():at]


@pytest.mark.parametrize("file", ["lt_build.cu", "radix_sort.cu"])
def test_waiting_kernels_use_no_read_only_loads(file):
    source = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, file)).read())
    waiting, helpers = [], {}
    for names, head, body in functions(source):
        if "__global__" in head:
            if "grid_wait()" in body:
                waiting.append((head, body))
        else:
            helpers[names[-1]] = (head, body)
    assert len(waiting) >= 4
    for head, body in waiting:
        seen, todo = set(), [(head, body)]
        while todo:  # the kernel and every helper that it reaches
            h, b = todo.pop()
            assert not re.search(r"const [\w:]+\s*\*\s*__restrict__", h), h
            assert "__ldg(" not in b, h
            for name in set(re.findall(r"(\w+)(?:<[^;<>()]*>)?\s*\(", b)) & set(helpers) - seen:
                seen.add(name)
                todo.append(helpers[name])
        # Before the wait only declarations of shared memory.
        before = [s.strip() for s in body.split("grid_wait()")[0].split(";")]
        assert all(not s or s.startswith(("__shared__", "extern __shared__", "constexpr")) for s in before), before
