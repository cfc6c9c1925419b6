"""Properties of the kernels' source that no run shows unless something has already gone wrong."""

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpu_ragged_dot_b200", "csrc")


def _code(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_roles_give_up_as_whole_warps():
    """Every role runs as whole warps and has warp-wide steps (votes, __syncwarp, tcgen05.ld) behind its waits.  A
    bounded wait whose result may differ between lanes would split the warp when it runs out, so barriers are waited
    for through mbar_wait_warp, and flags under a vote or with a block barrier behind."""
    kernels = [n for n in sorted(os.listdir(CSRC)) if n.startswith("rd_") and n.endswith(".cuh") and n != "rd_ptx.cuh"]
    waits = 0
    for name in kernels:
        code = _code(name).replace("if constexpr (kOneThread) return mbar_wait(bar, parity, abort_ptr);", "")  # one thread
        assert not re.search(r"\bmbar_wait\s*(<[^>]*>)?\s*\(", code), f"{name}: a lane may leave its warp behind"
        waits += len(re.findall(r"\bmbar_wait_warp\s*(?:<[^>]*>)?\s*\(", code))
        for m in re.finditer(r"\bwait_flag_ge\s*\(", code):
            voted = code[:m.start()].rstrip().endswith("__all_sync(0xffffffffu,")
            assert voted or re.match(r"[^;]*;\s*__syncthreads\(\)", code[m.start():]), name
    assert waits > 20
    assert "__all_sync(0xffffffffu, mbar_wait<kClusterScope>(bar, parity, ctl))" in _code("rd_ptx.cuh")
