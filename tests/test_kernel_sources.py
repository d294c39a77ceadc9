"""Rules for kernels that no run shows to be kept, read from the sources."""
import os
import re

CSRC = os.path.join(os.path.dirname(__file__), "..", "purhie_b200", "csrc")


def _code(path):
    with open(path) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_tensor_maps_in_memory_are_acquired_before_their_use():
    """A map is a kernel's __grid_constant__ parameter, or lies in global memory, where a copy from the host wrote it; then the
    kernel fences the map's proxy in front of the first prefetch or load that names it."""
    copying = 0
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith(".cu"):
            continue
        code = _code(os.path.join(CSRC, name))
        if "CUtensorMap" not in code:
            continue
        for kernel in re.split(r"__global__", code)[1:]:
            kernel = kernel[:kernel.find("\n}")]
            passed = kernel[:kernel.find("{")].count("__grid_constant__ CUtensorMap") + kernel[:kernel.find("{")].count("__grid_constant__ const CUtensorMap")
            uses = [m.start() for m in re.finditer(r"prefetch\.tensormap|\bload_\w+\(", kernel)]
            if passed or "CUtensorMap" not in kernel:
                continue
            copying += 1
            assert uses and 0 <= kernel.find("acquire_map(") < min(uses), name
        if "acquire_map(" in code:
            assert "fence.proxy.tensormap::generic.acquire" in code, name
    assert copying == 1
