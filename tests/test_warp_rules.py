"""The rules by which persistent warps size their work (warp_rules.h), run on
the host: the refill keys keep their whole range for full warps, and a spread
queue covers its rays."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cuda = "/usr/local/cuda"
    if not os.path.isdir(os.path.join(cuda, "include")) or not shutil.which("g++"):
        pytest.skip("needs g++ and the CUDA headers")
    out = tmp_path_factory.mktemp("warp_rules") / "libwarp_rules.so"
    subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-I", os.path.join(cuda, "include"),
                    "-I", os.path.join(ROOT, "photon_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "native", "warp_rules_test.cpp"), "-o", str(out)], check=True)
    lib = C.CDLL(str(out))
    for f in ("wr_lanes_for", "wr_refill_lanes", "wr_brief_lanes"):
        getattr(lib, f).restype = C.c_uint32
        getattr(lib, f).argtypes = [C.c_uint32, C.c_uint32]
    return lib


def test_full_warps_refill_where_the_key_says(lib):
    """Every value of trace_refill and vol_refill (1..32) holds as it is."""
    assert [lib.wr_refill_lanes(k, 32) for k in range(1, 33)] == list(range(1, 33))


@pytest.mark.parametrize("per_warp", [1, 2, 4, 8, 16])
def test_spread_warps_refill_at_half_of_their_rays(lib, per_warp):
    half = max(per_warp // 2, 1)
    assert [lib.wr_refill_lanes(k, per_warp) for k in range(1, 33)] == [min(k, half) for k in range(1, 33)]


@pytest.mark.parametrize("warps", [1, 2, 3, 152, 4864, 9728])
def test_spread_queues_are_covered(lib, warps):
    half = max(warps // 2, 1)
    for n in [0, 1, half - 1, half, half + 1, 2 * half, 16 * half, 16 * half + 1, 31 * half, 32 * half, 10 ** 7]:
        k = lib.wr_lanes_for(max(n, 0), warps)
        assert k in (1, 2, 4, 8, 16, 32)
        assert k == 32 or k * half >= n      # half of the warps hold the whole queue
        assert k == 1 or (k // 2) * half < n  # with no more lanes than that takes


@pytest.mark.parametrize("warps", [1, 2, 64, 2432, 9728])
def test_short_calls_are_all_in_flight(lib, warps):
    """Rays go by the warps' places only while half of the grid (what is
    resident) holds them all, and never with 16 lanes of a warp on."""
    half = max(warps // 2, 1)
    for n in [1, half, half + 1, 2 * half, 4 * half, 8 * half, 8 * half + 1, 16 * half, 16 * half + 1, 32 * half]:
        k = lib.wr_brief_lanes(n, warps)
        assert k in (1, 2, 4, 8, 32)
        assert k * half >= n
        assert k == 32 or k == 1 or (k // 2) * half < n
    for n in [32 * half + 1, 64 * half - 1, 64 * half, 2 ** 30]:
        assert lib.wr_brief_lanes(n, warps) == 0
