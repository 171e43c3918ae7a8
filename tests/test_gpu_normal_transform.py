"""The drive's own division and square root give the intrinsics' bits for every float that the
polar method can hand them: s in [2^-48, 1), all 402,653,184 values.  The bit-exactness of every
step kernel rests on it."""
import ctypes as C
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_every_float(tmp_path):
    import os
    from gpu4snn_gb300 import build
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native", "normal_transform.cu")
    lib = str(tmp_path / "normal_transform.so")
    r = subprocess.run([build.nvcc()] + build.NVCC_FLAGS + ["-shared", src, "-o", lib, "-cudart", "static"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    first, last = (int(np.float32(x).view(np.uint32)) for x in (2.0 ** -48, 1.0))
    out = (C.c_ulonglong * 4)()
    assert C.CDLL(lib).sweep_normal_transform(C.c_uint(first), C.c_uint(last), out) == 0
    assert out[3] == last - first == 402_653_184
    assert list(out[:3]) == [0, 0, 0]
