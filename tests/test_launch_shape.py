"""The transport's launch shape (csrc/cl_launch.h, compiled here for the host):
what cl_set_launch asks for is what is launched, also for few photons, and only
what is automatic follows the number of photons."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SMS = 148


@pytest.fixture(scope="module")
def shape(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("launch") / "launch_shape_check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-o", exe,
                    os.path.join(ROOT, "tests", "cpp", "launch_shape_check.cpp")], check=True)

    def call(n, resident, ctas=0, threads=0, chunk=0):
        args = [str(v) for v in (n, SMS, resident, ctas, threads, chunk)]
        out = subprocess.run([exe] + args, check=True, capture_output=True, text=True).stdout
        return tuple(int(v) for v in out.split())
    return call


@pytest.mark.parametrize("n", [1, 100, 2000, 37_887, 37_888, 10**6])
@pytest.mark.parametrize("ctas,threads,chunk", [(0, 256, 0), (0, 192, 0), (0, 128, 0), (0, 64, 0), (0, 32, 0),
                                                (1, 256, 0), (1, 128, 0), (2, 64, 0), (1, 0, 0), (3, 0, 32),
                                                (4, 256, 256), (0, 0, 64)])
def test_what_is_asked_for_is_launched(shape, n, ctas, threads, chunk):
    resident = 8 if threads in (32, 64, 128) else 4
    grid, t, c = shape(n, resident, ctas, threads, chunk)
    if threads:
        assert t == threads
    elif ctas:
        assert t == 256
    if chunk:
        assert c == chunk
    per_sm = min(ctas or resident, resident)
    assert 1 <= grid <= SMS * per_sm
    assert c >= 1 and (grid - 1) * (t // 32) * c < n         # no CTA without a first chunk
    if not chunk:
        # every photon of a small launch has a warp of its own where the warps suffice, no
        # warp has more than eight warps per SM would leave it
        warps = SMS * per_sm * (t // 32)
        assert c <= max(32, -(-n // min(warps, 8 * SMS)))


@pytest.mark.parametrize("n,want", [
    # few photons: 128 threads, spread over eight warps per SM (or one photon per warp)
    (1, (1, 128, 1)), (100, (25, 128, 1)), (1184, (296, 128, 1)), (1185, (149, 128, 2)), (2000, (250, 128, 2)),
    (37_887, (296, 128, 32)),
    # more: 256 threads, whole warps' chunks of 32 to 256
    (37_888, (148, 256, 32)), (10**6, (592, 256, 32)), (4 * 10**6, (592, 256, 32)), (10**7, (592, 256, 128)),
    (10**9, (592, 256, 256))])
def test_automatic_shapes(shape, n, want):
    assert shape(n, 4) == want
