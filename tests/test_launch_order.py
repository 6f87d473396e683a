"""A kernel that lets its successor start before it has its tensor-memory columns can wait for ever: the successor's CTA may take the columns and then
wait (griddepcontrol.wait) for the kernel whose CTA waits for them.  Read from the sources: in every kernel that allocates tensor memory,
launch_dependents stands behind the allocation and the barrier that follows it."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "nano-vllm-rs_b200" / "csrc"


def _kernels(path):
    """Source text from one __global__ to the next."""
    text = re.sub(r"//[^\n]*", "", path.read_text())
    return text.split("__global__")[1:]


def test_dependents_start_behind_the_tensor_memory_allocation():
    found = 0
    for path in sorted(CSRC.glob("*.cu")):
        for body in _kernels(path):
            alloc = re.search(r"\btmem_alloc(_cg2)?<", body)
            if alloc is None:
                continue
            found += 1
            barrier = re.compile(r"__syncthreads\(\)|cluster_sync_all\(\)").search(body, alloc.end())
            starts = [m.start() for m in re.finditer(r"pdl_launch_dependents\(\)", body)]
            assert starts and min(starts) > barrier.end(), f"{path.name}: successors start before the columns are there"
    assert found >= 5
