"""Errors of a cluster launch, on a host without a GPU: reported as themselves, every time."""
import ctypes
import os

import pytest

from rochpl_b200 import build


@pytest.mark.parametrize("kind", ["d", "f"])
def test_error_is_its_own_and_not_kept(kind):
    """The first failing launch used to mark the cluster size as one that the GPU has no
    place for, and every later call of the process returned cudaErrorLaunchFailure."""
    import torch

    if torch.cuda.is_available():
        pytest.skip("needs a host without a GPU")
    lib = ctypes.CDLL(build.LIB) if os.path.exists(build.LIB) else ctypes.CDLL(build.build())
    f = lib[f"_ZN4hplb25launch_unit_lower_inverseI{kind}EE9cudaErrorPKT_liS4_PS2_lP11CUstream_stPi"]
    P, q, i = ctypes.c_void_p, ctypes.c_int64, ctypes.c_int
    f.argtypes = [P, q, i, P, P, q, P, P]
    codes = [f(None, 64, 64, None, None, 64, None, None) for _ in range(2)]
    assert codes[0] == codes[1] and codes[0] not in (0, 719), codes
