"""The landmark refresh's index checks, which come before anything of the context is used and so run without a
GPU (the context pointer stands for one): the first bad index in track order decides the message, whatever the
number of intrinsics and with it of the chunks the checks run in, and a chunk's flags are not what the call
spends its memory on where there are more intrinsics than a chunk has entries."""
import os
import subprocess
import sys

import pytest

_CALL = """
import ctypes as C, resource, sys
import numpy as np
from openmvg_ba_cuda import abi
from openmvg_ba_cuda._lib import lib

n, intrinsics = int(sys.argv[1]), int(sys.argv[2])
p = lambda a, t: a.ctypes.data_as(C.POINTER(t))
pose, intrinsic = np.zeros(n, np.uint32), np.zeros(n, np.uint32)
for at, what in [(int(a), w) for a, w in (s.split(":") for s in sys.argv[3:])]:
    (pose if what == "pose" else intrinsic)[at] = 1 if what == "pose" else intrinsics
keep = (np.ones(3 * n), np.ones(n, np.uint8), np.arange(n + 1, dtype=np.uint64), np.ones(2 * n), np.ones(n, np.uint8),
        np.ones(n, np.uint8), np.ones(n), np.ones(n, np.uint8))
points, active, offset, pixel, support, update, error, out = keep
tracks = abi.LandmarkTracks(n, p(points, C.c_double), p(active, C.c_uint8), p(offset, C.c_uint64),
                            p(pose, C.c_uint32), p(intrinsic, C.c_uint32), p(pixel, C.c_double), p(support, C.c_uint8))
result = abi.RefreshResult(p(update, C.c_uint8), p(error, C.c_double), p(out, C.c_uint8), 0, 0)
cams = (abi.Intrinsic * intrinsics)()
context, err = C.create_string_buffer(1024), abi.Error()
before = resource.getrusage(resource.RUSAGE_SELF).ru_maxrss
code = lib().omvgba_sfm_refresh_reprojection(C.cast(context, C.c_void_p), 1, (abi.Pose * 1)(), intrinsics, cams,
                                             C.byref(tracks), C.byref(result), C.byref(err))
print(code, (resource.getrusage(resource.RUSAGE_SELF).ru_maxrss - before) * 1024, err.message.decode())
"""


def _refresh(*args):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, PYTHONPATH=os.path.join(root, "openmvg-rs_b200"))
    out = subprocess.run([sys.executable, "-c", _CALL, *map(str, args)], env=env, check=True, capture_output=True, text=True)
    code, grown, message = out.stdout.strip().split(" ", 2)
    return int(code), int(grown), message


@pytest.mark.parametrize("observations,intrinsics", [(1000, 4), (262_145, 4), (300_000, 150_000), (300_000, 2_000_000)])
def test_the_first_bad_index_decides(observations, intrinsics):
    from openmvg_ba_cuda import abi
    half, last = observations // 2, observations - 1
    assert _refresh(observations, intrinsics, f"{last}:pose", f"{half}:intrinsic")[::2] == (
        abi.OMVGBA_INVALID_PROBLEM, "track intrinsic index out of range")
    code, grown, message = _refresh(observations, intrinsics, f"{last}:intrinsic", f"{half}:pose")
    assert (code, message) == (abi.OMVGBA_INVALID_PROBLEM, "track pose index out of range")
    assert grown <= (8 << 20) + 2 * intrinsics  # one chunk's flags and some thread stacks, not 64 chunks' flags
