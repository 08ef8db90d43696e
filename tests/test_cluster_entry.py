"""A block of a cluster may reach into another's shared memory only once that
block is known to run: in every kernel a cluster barrier stands before the
first use of a mapped address.  (Read from the source: the early access is a
race that no run need show.)"""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "itensornumericalanalysis.jl_gb300" / "csrc"


def test_barrier_before_first_remote_access():
    seen = 0
    for src in sorted(CSRC.glob("*.cu*")):
        text = re.sub(r"//[^\n]*", "", src.read_text())
        for kernel in re.split(r"__global__", text)[1:]:
            body = kernel[: kernel.find("\n}\n")]
            if "map_shared_rank" not in body:
                continue
            seen += 1
            first = body.index("map_shared_rank")
            barrier = re.search(r"\bcl\.sync\(\)|this_cluster\(\)\.sync\(\)", body)
            assert barrier and barrier.start() < first, src.name + kernel[:80]
    assert seen > 0
