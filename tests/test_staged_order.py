"""Order of the tensor-memory accesses of the staged z pass, read from its source: the allocation
and the release by one warp are separated from the other warps' accesses by a block barrier between
tcgen05.fence::before_thread_sync and ::after_thread_sync, as the PTX memory model asks."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _kernel():
    with open(os.path.join(ROOT, "spns_b200", "csrc", "zpass_staged.cuh")) as fh:
        src = re.sub(r"//[^\n]*", "", fh.read())
    return src[src.index("k3_rot_staged(Geo g"):]


def test_allocation_and_release_are_fenced():
    body = _kernel()
    names = r"tmem_alloc|tmem_free|tmem_st4|tmem_ld4|tmem_wait_ld|tmem_wait_st|tmem_fence_before_sync|tmem_fence_after_sync|__syncthreads|block_max4"
    calls = re.findall(r"\b(" + names + r")\b\s*[<(]", body)
    assert calls[:5] == ["tmem_alloc", "tmem_fence_before_sync", "__syncthreads", "tmem_fence_after_sync", "tmem_st4"]
    assert calls[-5:] == ["tmem_wait_ld", "tmem_fence_before_sync", "block_max4", "tmem_fence_after_sync", "tmem_free"]
