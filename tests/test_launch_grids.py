"""A persistent or cooperative grid is sized by the occupancy of the kernel that
it launches, not of another one: read from the launchers' source, since no
result depends on it."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "photon_gb300", "csrc")


def _text(name):
    return open(os.path.join(CSRC, name)).read()


def test_adjoint_resolve_has_its_own_grid():
    cu, host = _text("adjoint.cu"), _text("renderer.cpp")
    grid, threads = re.search(r"k_adj_resolve<<<([^,]+), (\w+),", cu).groups()
    assert grid == "blocks"
    assert re.search(r"__launch_bounds__\(%s\) k_adj_resolve\b" % threads, cu)
    own = re.search(r"int (\w+)\(\) \{ return resident_blocks\(k_adj_resolve, %s\); \}" % threads, cu).group(1)
    passed = re.search(r"launch_adj_resolve\((\w+),", host).group(1)
    assert re.search(r"const int %s = r->sm_count \* %s\(\);" % (passed, own), host)


def test_clustering_grid_is_that_of_the_launched_kernel():
    """A cooperative launch of more blocks than are resident fails, so the
    occupancy asked for must be that of the radius' own kernel."""
    cu = _text("bvh_gpu.cu")
    launched = re.search(r"cudaLaunchCooperativeKernel\((\w+), dim3\(ploc_blocks\)", cu).group(1)
    assert re.search(r"device_limits\(%s\)" % launched, cu)
    asked = re.findall(r"cudaOccupancyMaxActiveBlocksPerMultiprocessor\(&d\.ploc_blocks, ([^,]+),", cu)
    argument = re.search(r"DeviceLimits device_limits\(const void \*(\w+)\)", cu).group(1)
    assert asked == [argument]
