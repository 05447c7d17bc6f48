"""Order of the steps in a kernel's start, read from the sources.

A kernel that allocates tensor memory may let the next kernel's CTAs onto its SM (programmatic dependent launch) only when the whole CTA
knows that the allocation is done: the trigger of any one thread counts for its CTA, and two kernels that each hold a part of an SM's 512
columns and wait for the rest would never end."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "distributed_inference_server_b200", "csrc")


def kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        s = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__", s):
            name = re.search(r"(\w*kernel\w*)\s*\(", s[m.start():])
            at = m.start() + name.end()
            depth = 1
            while depth:  # the end of the parameter list
                depth += {"(": 1, ")": -1}.get(s[at], 0)
                at += 1
            start = at = s.index("{", at)
            depth = 0
            while True:
                depth += {"{": 1, "}": -1}.get(s[at], 0)
                at += 1
                if depth == 0:
                    break
            yield name.group(1), s[start:at]


def test_tensor_memory_is_allocated_before_the_next_kernel_may_start():
    seen = 0
    for name, body in kernels():
        alloc = re.search(r"tmem_alloc|tcgen05\.alloc", body)
        trigger = body.find("pdl_launch_dependents")
        if alloc is None or trigger < 0:
            continue
        seen += 1
        barrier = body.find("__syncthreads()", alloc.end())
        assert 0 <= barrier < trigger, f"{name}: the trigger stands in front of the barrier that follows the allocation"
    assert seen >= 3


def test_shared_memory_of_other_ctas_is_written_only_when_they_run():
    """CTAs of a cluster are placed together, but only a cluster barrier says that the others have begun: it stands in front of the first
    store into their shared memory (st.shared::cluster, by itself or in a helper)."""
    store = re.compile(r"st\.shared::cluster|\bst_cluster\s*\(|\bswap\s*\(\s*s\b")
    waits = re.compile(r"barrier\.cluster\.wait|\bcluster_wait\s*\(|\bcluster_sync(_all)?\s*\(")
    seen = 0
    for name, body in kernels():
        first = store.search(body)
        if first is None:
            continue
        seen += 1
        wait = waits.search(body)
        assert wait is not None and wait.start() < first.start(), f"{name}: stores into another CTA's shared memory before it is known to run"
    assert seen >= 2


def test_empty_slices_leave_the_stages_alone():
    """Layer-list attention zeroes the padding columns of its key stages at its start and lays the warps' states over the stages at its end.  The
    barriers in between are those of the key tiles: a slice without a key has none, so it must not write the columns either."""
    body = dict(kernels())["stack_attn_mma_kernel"]
    zero = re.search(r"if\s*\(([^;{]*)\)\s*for\s*\([^;]*;[^;]*;[^)]*\)\s*Ks\[[^;]*\]\s*=\s*0;", body)
    assert zero is not None and zero.start() < body.find("__syncthreads()")
    assert "k_end > k_begin" in zero.group(1)
