"""Kernels of a launch chain start while the kernel before still writes their operands: what they read of those is not declared as
standing still (``__restrict__``), in the source at least, which is what the compiler goes by."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "csrc")
# read, and written by no kernel of a chain: weights and a batch's tables
STILL = {"w", "b", "bias", "last_token", "tok_seq", "tok_pos", "block_tables"}
# written only
RESULTS = {"y", "res_out", "mean_out", "rstd_out", "out"}


def _kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        for body in re.split(r"\n__global__", open(path).read())[1:]:
            name = re.search(r"(\w+_kernel)\s*\(", body)
            head, _, rest = body[name.start():].partition(") {\n")
            yield name.group(1), head, re.split(r"\n}\n", rest)[0]


def test_moving_operands_are_plain_pointers():
    seen = set()
    for name, head, body in _kernels():
        if "chain_wait()" not in body:
            continue
        seen.add(name)
        for const, param in re.findall(r"(const )?[\w:]+\s*\*\s*__restrict__\s+(\w+)", head):
            assert param in (STILL if const else RESULTS), (name, param)
            if not const:                                  # a result: no load through it
                assert not re.search(r"(ld8<T>\(|= )" + param + r"\b", body), (name, param)
    assert {"norm_fwd_kernel", "gated_fwd_kernel", "logits_gather_kernel", "kv_rotary_blocked_kernel", "paged_decode_kernel",
            "gemm_skinny_kernel"} <= seen
