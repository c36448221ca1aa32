"""Which kernels may let the next one start before they have waited for the one before (csrc/common.cuh, chain_next): never those
that run right ahead of a GEMM, which reads the group offsets before its own wait, and none of the expert-parallel exchange."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ateniaengine_b200", "csrc")

# ahead of one of these kernels comes no writer of offsets that a GEMM behind could read too early: routers, sorts (the gather or
# the digits follow), a layer's last kernels, and between two GEMMs the adder of split tiles
EARLY = {"router_dmma_direct_kernel", "router_splitk_kernel", "dispatch_small_kernel", "dispatch_cluster_kernel", "combine_kernel",
         "grouped_gemv_kernel", "rmsnorm_rows_kernel", "decode_splitk_reduce_kernel"}


def kernels():
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        text = re.sub(r"//.*", "", open(path, encoding="utf-8").read())
        for part in text.split("__global__")[1:]:
            body = part[part.index("{"):]
            end, depth = 0, 0
            for end, c in enumerate(body):
                depth += (c == "{") - (c == "}")
                if depth == 0:
                    break
            name = re.findall(r"(\w+)\s*\(", re.sub(r"__\w+__\s*\([^)]*\)", "", part[:part.index("{")]))[0]
            yield os.path.basename(path), name, body[:end]


def test_only_known_kernels_start_the_next_one_early():
    early, chained = set(), 0
    for path, name, body in kernels():
        nexts, waits = body.find("chain_next()"), body.find("chain_wait()")
        assert path != "ep.cu" or (nexts < 0 and waits < 0), name
        chained += waits >= 0
        if nexts >= 0 and "if (between) chain_next();" not in body and (waits < 0 or nexts < waits):
            early.add(name)
    assert early == EARLY and chained >= 12


def test_the_kernels_ahead_of_a_gemm_wait_first():
    seen = set()
    for _, name, body in kernels():
        if name in ("gather_rows_kernel", "quantize_digits_kernel"):
            body = body.replace("if (between) chain_next();", "")
            assert 0 <= body.index("chain_wait()") < body.index("chain_next()")
            seen.add(name)
    assert len(seen) == 2


def test_the_exchange_launches_plainly():
    text = open(os.path.join(CSRC, "ep.cu"), encoding="utf-8").read()
    assert "launch_chained" not in text and "<<<" in text
