"""A wait that gives up must not leave the rest of its CTA behind.  Read from the source, since no GPU is made to hang for it: a warp
leaves its work early only as a whole, and never one that meets others at a named barrier."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "csrc")
FILES = sorted(p for p in glob.glob(os.path.join(CSRC, "*.cu*")) if not p.endswith("sxb_common.cuh"))


def test_warps_leave_as_a_whole():
    """The result of a wait is used after a vote, or not at all."""
    seen = 0
    for path in FILES:
        lines = [line.split("//")[0] for line in open(path).read().split("\n")]
        for line, behind in zip(lines, lines[1:]):
            if "mbar_wait_to(" not in line:
                continue
            seen += 1
            result = re.search(r"const bool (\w+) = mbar_wait_to\(", line)
            assert ("__all_sync(0xffffffffu, mbar_wait_to(" in line or "&& prof)" in line          # (only times the wait)
                    or result and f"__all_sync(0xffffffffu, {result.group(1)})" in behind), (path, line)
    assert seen > 40


def test_no_warp_of_a_named_barrier_leaves_early():
    kernels = 0
    for path in FILES:
        for body in re.split(r"\n__global__", open(path).read())[1:]:
            body = body.split("\n}\n")[0]
            at = [m.start() for m in re.finditer(r"named_bar_sync8?\(|bar\.sync 1, ", body)]
            if not at or "mbar_wait" not in body:
                continue
            kernels += 1
            # the branch of the warps that meet: the last one of the kernel
            branch = body[body.rfind("\n  } else {\n", 0, at[0]): body.find("\ndone:")]
            assert branch.count("mbar_wait_on(") >= 1 and "goto done" not in branch and "return;" not in branch, path
    assert kernels == 6
