"""A kernel lets its successor in the stream start early only once it holds its tensor memory: a successor that took the columns
first and then waited for this grid would never end."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "csrc")


def test_tensor_memory_is_taken_before_dependents_may_start():
    seen = set()
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        for body in re.split(r"\n__global__", open(path).read())[1:]:
            at = min((i for i in (body.find("griddepcontrol.launch_dependents"), body.find("chain_next()")) if i >= 0), default=-1)
            if at < 0 or "tmem_alloc(" not in body.split("\n}\n")[0]:
                continue
            seen.add(re.search(r"(\w+_kernel)\s*\(", body).group(1))
            alloc = body.find("tmem_alloc(")
            assert alloc < at, path
            between = body[alloc:at]
            assert "__syncthreads()" in between or "cluster_sync_all()" in between, path
    assert {"attn_bwd_dq_kernel", "attn_bwd_dq128_kernel", "gemm_skinny_kernel"} <= seen
