"""Entry points of the kernel library with arguments that leave nothing to do: host code, checked without a GPU (the launch
itself may answer with an error here; the process must not end)."""
import subprocess
import sys

import pytest

from tinyinfinitrain_b200._build import KERNEL_LIB


def _run(call):
    code = f"""
import ctypes
lib = ctypes.CDLL({str(KERNEL_LIB)!r})
null, f = None, ctypes.c_float
print("rc", {call})
"""
    return subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120)


@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("B,T,H,hd", [(2, 3, 0, 64), (2, 3, 4, 0), (0, 3, 4, 64), (2, 0, 4, 64)])
def test_rope_of_nothing(B, T, H, hd, dtype):
    r = _run(f"lib.titb_rope_strided(null, null, {B}, {T}, {H}, {hd}, ctypes.c_longlong(64), 0, f(1e4), 0, {dtype}, null)")
    assert r.returncode == 0 and "rc 0" in r.stdout, (r.returncode, r.stdout, r.stderr[-500:])
