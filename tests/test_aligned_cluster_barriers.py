"""`barrier.cluster.*.aligned` is undefined unless all lanes of a warp execute it together: in every kernel source the
statement before one is a reconvergence (or another such barrier), so none relies on where the compiler joins the lanes
of a loop or a branch."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ateniaengine_b200", "csrc")
JOINED = re.compile(r"__syncwarp\(\);|__syncthreads\(\);|barrier\.cluster\.(arrive|wait)\.[a-z.]*aligned;")


def test_every_aligned_cluster_barrier_follows_a_reconvergence():
    seen = 0
    for path in glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")):
        lines = [re.sub(r"//.*", "", line).strip() for line in open(path, encoding="utf-8")]
        lines = [line for line in lines if line]
        for i, line in enumerate(lines):
            if re.search(r"barrier\.cluster\.(arrive|wait)\.[a-z.]*aligned", line):
                seen += 1
                assert JOINED.search(lines[i - 1]), (os.path.basename(path), lines[i - 1], line)
    assert seen >= 6
