"""A shared array that is read or written as vectors asks for their alignment; where the linker happens to put it is not one."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ateniaengine_b200", "csrc")
CAST = re.compile(r"reinterpret_cast<(?:const )?(?:float4|uint4|int4|double2|float2|uint2)\*>\(&?(\w+)\[")
PLAIN = r"__shared__ (?:float|double|int|int32_t|uint8_t|uint16_t|uint32_t|unsigned char) (?:\w+(?:\[[^;,]*\])*, )*%s\["


def test_vector_accesses_to_shared_arrays_are_aligned():
    seen = 0
    for path in glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")):
        text = re.sub(r"//.*", "", open(path, encoding="utf-8").read())
        kernels = re.split(r"__global__", text)
        for kernel in kernels:
            for name in set(CAST.findall(kernel)):
                seen += bool(re.search(r"__shared__ __align__\(16\) \w+ %s\[" % name, kernel))
                assert not re.search(PLAIN % name, kernel), (os.path.basename(path), name)
    assert seen >= 1
