"""Orderings inside kernels that no run on a GPU can be relied on to show, checked in the source."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "infmoe_b200", "csrc")


def _signatures():
    """(file, name, parameter list, body) of every __global__ function, comments removed."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        with open(path) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for m in re.finditer(r"__global__[^;{]*?(\w+)\s*\(", text):
            if m.group(1) == "__launch_bounds__":
                m = re.compile(r"\)\s*(\w+)\s*\(").search(text, m.end())
            start = text.index("{", m.end())
            depth, i = 0, start
            while True:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
                if depth == 0:
                    break
            yield os.path.basename(path), m.group(1), text[m.end():start], text[start:i]


def _kernels():
    return [(file, name, body) for file, name, _, body in _signatures()]


def test_kernels_are_found():
    names = {name for _, name, _ in _kernels()}
    assert {"route_small_kernel", "dispatch_kernel", "ffn_umma_kernel", "gather_kernel"} <= names


@pytest.mark.parametrize("file,name,body", [k for k in _kernels() if re.search(r"map_shared_rank|leader_addr\(", k[2])],
                         ids=lambda v: v if len(v) < 40 else "")
def test_other_blocks_memory_is_touched_only_behind_a_cluster_barrier(file, name, body):
    """Distributed shared memory may be accessed once the target block is known to have started, which only a
    cluster-wide barrier establishes."""
    remote = re.search(r"map_shared_rank|leader_addr\(", body).start()
    barrier = re.search(r"cluster\.sync\(\)|cluster_sync\(\)|barrier\.cluster\.wait", body)
    assert barrier and barrier.start() < remote, f"{file}: {name} reaches another block's memory before any cluster barrier"


def test_sums_of_a_cut_tile_are_read_behind_a_warp_barrier():
    """Lane 0 counts the arrivals and fences; a shuffle hands the count to the other lanes but orders no memory, so a
    warp barrier has to stand between it and their reads of what other blocks stored."""
    body = next(b for _, n, b in _kernels() if n == "ffn_umma_kernel")
    counted, read = body.index("atomicAdd(counter"), body.index("__ldcg(src")
    handed_on = body.rindex("__shfl_sync(0xffffffffu, done", counted, read)
    assert "__threadfence();" in body[counted:handed_on]
    assert "__syncwarp();" in body[handed_on:read]


@pytest.mark.parametrize("file,name,params,body", [k for k in _signatures() if "pdl_wait" in k[3]],
                         ids=lambda v: v if len(v) < 40 else "")
def test_kernels_that_start_early_promise_nothing_about_what_others_still_write(file, name, params, body):
    """A kernel that starts before its predecessor has ended may not read what that one writes through the read-only path:
    `const T* __restrict__` parameters and __ldg promise that nobody writes during the kernel, and a load under that promise
    may be moved above the wait."""
    assert not re.search(r"const\s+\w+\s*\*\s*__restrict__", params), f"{file}: {name}"
    for load in re.findall(r"__ldg\((?:[^()]|\([^()]*\))*\)", body):
        assert re.search(r"\b(scales|bound)\b", load), f"{file}: {name}: {load}"      # of the weights, written before any pass


@pytest.mark.parametrize("file,name,body", [k for k in _kernels() if re.match(r"route_|dispatch_|scatter_", k[1]) and "pdl_wait" in k[2]],
                         ids=lambda v: v if len(v) < 40 else "")
def test_kernels_before_the_gemms_let_their_successor_start_after_their_own_wait(file, name, body):
    """Their successors read, before their own wait, what was complete when this kernel's wait ended."""
    assert body.index("pdl_wait()") < body.index("pdl_trigger()"), f"{file}: {name}"
